"""C entries that the package's own engines no longer take, numerically: the FP64
FMA transform, the FP64 DCT rows, the double plans without sliced products, and
the single passes that fused ones replaced."""
import ctypes

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def dev(a):
    return torch.tensor(np.ascontiguousarray(a), device="cuda")


def rel(a, b):
    return float(np.linalg.norm(a - b) / np.linalg.norm(b))


@pytest.mark.parametrize("nr,nz", [(3, 5), (33, 31), (64, 128), (130, 257)])
def test_fma_transform(nr, nz):
    from pyaxisymflow_gb300 import _native as N
    rng = np.random.default_rng(nr)
    Er, Ei = rng.standard_normal((2, nr, nr))
    EzinvT, EzT = rng.standard_normal((2, nz, nz))
    inv, w = rng.standard_normal((2, nr, nz))
    wide = dev(rng.standard_normal((nr, nz + 3)))
    wide[:, 1:nz + 1] = dev(w)
    out, work = dev(np.zeros((nr, nz + 2))), dev(np.zeros(2 * nr * nz))
    t = [dev(x) for x in (Ei, EzinvT, inv, Er, EzT)]
    N.call("axi_fd_transform_f64", N.ptr(out), nz + 2, ctypes.c_void_p(wide.data_ptr() + 8),
           nz + 3, *(N.ptr(x) for x in t), N.ptr(work), nr, nz, N.stream_of(out))
    got = out.cpu().numpy()
    ref = Er @ (((Ei @ (w @ EzinvT)) * inv) @ EzT)
    # four products of up to max(nr, nz) terms, sums of random sign
    assert rel(got[:, :nz], ref) < 4 * max(nr, nz) * 2.0 ** -53
    assert not got[:, nz:].any()


@pytest.mark.parametrize("rows,N_", [(1, 2), (5, 6), (33, 48), (7, 162), (20, 1024), (9, 1536),
                                     (3, 2048)])
def test_dct_rows_in_double(rows, N_):
    from pyaxisymflow_gb300 import _native as N
    from pyaxisymflow_gb300.engine import cosine_basis, dct_table
    x = np.random.default_rng(N_).standard_normal((rows, N_))
    basis, table = cosine_basis(N_), dev(dct_table(N_, np.float64))
    for forward, want in ((1, x @ basis.T), (0, x @ basis)):
        src, out = dev(x), dev(np.zeros_like(x))
        plan = torch.empty(int(N.lib().axi_dct64_plan_bytes(rows, N_)), dtype=torch.uint8,
                           device="cuda")
        s = N.stream_of(out)
        N.call("axi_dct64_plan_f64", N.ptr(src), N.ptr(out), rows, N_, N.ptr(table), forward,
               N.ptr(plan), s)
        N.call("axi_dct64_run_f64", N.ptr(plan), rows, N_, forward, s)
        # log2 N stages and the dense sum's own rounding
        assert rel(out.cpu().numpy(), want) < 8 * np.log2(2 * N_) * 2.0 ** -53


@pytest.mark.parametrize("M,N_,K", [(1, 1, 1), (65, 33, 17), (128, 256, 100)])
def test_dgemm(M, N_, K):
    from pyaxisymflow_gb300 import _native as N
    rng = np.random.default_rng(M)
    A, B, S = rng.standard_normal((M, K)), rng.standard_normal((K, N_)), rng.standard_normal(
        (M, N_))
    for scale in (None, S):
        c, a, b = dev(np.zeros((M, N_))), dev(A), dev(B)
        sd = dev(S) if scale is not None else None
        N.call("axi_dgemm_f64", N.ptr(c), N_, N.ptr(a), K, N.ptr(b), N_,
               N.ptr(sd) if sd is not None else None, M, N_, K, N.stream_of(c))
        want = A @ B if scale is None else (A @ B) * S
        assert rel(c.cpu().numpy(), want) < (K + 1) * 2.0 ** -53


PLAN_DENSE, PLAN_DCT_Z = 0, 2


@pytest.mark.parametrize("flags", [PLAN_DENSE, PLAN_DCT_Z])
@pytest.mark.parametrize("sediment", [False, True])
def test_double_plans_without_sliced_products(flags, sediment):
    """Two cases stepped by a plan of the FP64 FMA products, and one of FP64 DCTs
    around the radial ones, against the engine's own plan on the same bases."""
    from pyaxisymflow_gb300 import _native as N
    from pyaxisymflow_gb300 import engine as E
    cases = [E.RigidBodyCase(nz=96, nr=52, dx=2.0 / 96, r_sphere=0.2, z_cm=1.0, ramp=False,
                             U0=0.0 if sediment else 1.0, sediment=sediment, rho_s=2.0, seed=1),
             E.RigidBodyCase(nz=64, nr=32, dx=2.0 / 64, r_sphere=0.2, z_cm=1.2, ramp=False,
                             U0=0.0 if sediment else 1.0, sediment=sediment, rho_s=2.0, seed=2)]
    ref, ens = (E.RigidEnsemble(cases, precision="f64") for _ in range(2))
    tables = [dev(E.dct_table(c.nz, np.float64)) for c in cases]
    structs = (E.AxiCase * 2)()
    for k, m in enumerate(ens.members):
        structs[k] = m.struct
        structs[k].dct_table = tables[k].data_ptr()
    info, lib, s = E.AxiPlanInfo(), N.lib(), N.stream_of(tables[0])
    N.check(lib.axi_plan_init(ctypes.addressof(structs), 2, 8, flags, ctypes.byref(info)), "init")
    plan = torch.empty(int(info.bytes), dtype=torch.uint8, device="cuda")
    N.check(lib.axi_plan_upload(ctypes.addressof(structs), ctypes.byref(info),
                                ctypes.c_void_p(plan.data_ptr()), s), "upload")
    N.check(lib.axi_rigid_step_f64(ctypes.byref(info), ctypes.c_void_p(plan.data_ptr()), 5, s),
            "step")
    ref.step(5)
    torch.cuda.synchronize()
    for a, b in zip(ens.fields, ref.fields):
        for f in ("omega", "psi", "u_z", "u_r"):
            # a few 1e-15 a solve, five steps
            assert rel(a[f].cpu().numpy(), b[f].cpu().numpy()) < 1e-12, f
    np.testing.assert_allclose(ens.state.cpu().numpy()[:, :6], ref.state.cpu().numpy()[:, :6],
                               rtol=1e-11, atol=1e-13)


def test_passes_that_fused_ones_replaced():
    from pyaxisymflow_gb300 import _native as N
    rng = np.random.default_rng(5)
    nr, nz, dx, dt, G = 20, 37, 0.03, 0.01, 1.3
    n = nr * nz
    # sigma, then times chi, against both in one pass
    e1, e2 = rng.standard_normal((2, nr, nz))
    e1[:8, :9] = e2[:8, :9] = 0.0
    chi = np.where(rng.random((nr, nz)) < 0.3, 0.0, rng.random((nr, nz)))
    outs = []
    for fused in (False, True):
        sg = [dev(np.zeros((nr, nz))) for _ in range(3)]
        gr = [dev(np.zeros((nr, nz))) for _ in range(4)]
        a, b, c = dev(e1), dev(e2), dev(chi)
        s = N.stream_of(a)
        if fused:
            N.call("axi_soft_stress_f64", *(N.ptr(x) for x in sg), G, dx, N.ptr(a), N.ptr(b),
                   *(N.ptr(x) for x in gr), N.ptr(c), nr, nz, s)
        else:
            N.call("axi_solid_sigma_f64", *(N.ptr(x) for x in sg), G, dx, N.ptr(a), N.ptr(b),
                   *(N.ptr(x) for x in gr), nr, nz, s)
            N.call("axi_soft_stress_mask_f64", *(N.ptr(x) for x in sg), N.ptr(c), n, s)
        outs.append([x.cpu().numpy() for x in sg + gr])
    for a, b in zip(*outs):
        np.testing.assert_array_equal(a, b)
        np.testing.assert_array_equal(np.signbit(a), np.signbit(b))
    # particles moved, interpolated and copied back, against the one call
    Z, R = np.meshgrid((np.arange(nz) + 0.5) * dx, (np.arange(2 * nr) + 0.5) * dx)
    w, uz, ur = rng.uniform(-1, 1, (3, nr, nz))
    outs = []
    for fused in (False, True):
        zp, rp, vp, wd, Zd, Rd, uzd, urd = (dev(x) for x in (Z, R, 0 * Z, w, Z, R, uz, ur))
        work = torch.empty(int(N.lib().axi_p2m_mp4_work_bytes(2 * nr, nz)), dtype=torch.uint8,
                           device="cuda")
        s = N.stream_of(wd)
        if fused:
            N.call("axi_advect_particles_f64", *(N.ptr(x) for x in (zp, rp, vp, wd, Zd, Rd, uzd,
                                                                    urd)),
                   nr, nz, dx, dt, 0, N.ptr(work), s)
        else:
            full = dev(0 * Z)
            N.call("axi_advect_particles_prepare_f64", *(N.ptr(x) for x in (zp, rp, vp, wd, uzd,
                                                                            urd)), nr, nz, dt, s)
            N.call("axi_particles_to_mesh_2d_mp4_f64", N.ptr(zp), N.ptr(rp), N.ptr(vp),
                   N.ptr(full), 2 * nr, nz, dx, dx, 0, N.ptr(work), s)
            wd, zp, rp = full[nr:], Zd, Rd
        outs.append([x.cpu().numpy() for x in (wd, zp, rp, vp)])
    for a, b in zip(*outs):
        np.testing.assert_array_equal(a, b)
    # residual, then its split, against both in one pass
    psi, rhs, ar, az, wt = (rng.standard_normal(x) for x in ((nr, nz), (nr, nz), (nr, 3), (nz, 3),
                                                             nr))
    t = [dev(x) for x in (rhs, psi, wt, ar, az)]
    pair = [torch.empty(nr, nz, device="cuda") for _ in range(4)]
    res = torch.empty(nr, nz, dtype=torch.float64, device="cuda")
    s = N.stream_of(res)
    args = [N.ptr(x) for x in t] + [nr, nz, 0.7, -1.3, s]
    N.call("axi_fd_residual_f64", N.ptr(res), *args)
    N.call("axi_tc_split_f64", N.ptr(pair[0]), N.ptr(pair[1]), N.ptr(res), n, s)
    N.call("axi_fd_residual_split_f64", N.ptr(pair[2]), N.ptr(pair[3]), *args)
    assert torch.equal(pair[0], pair[2]) and torch.equal(pair[1], pair[3])
