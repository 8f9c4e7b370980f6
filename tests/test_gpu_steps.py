"""Full per-timestep loops on the GPU against the golden vectors and the oracle."""
import numpy as np
import pytest
import torch

from oracle import kernels as K
from oracle import simulation as sim

pytestmark = pytest.mark.gpu


def rel_l2(a, b):
    return float(np.linalg.norm(a - b) / max(np.linalg.norm(b), 1e-300))


def test_rigid_sphere_loop_against_golden(golden):
    from pyaxisymflow_gb300.simulation import RigidSphereSimulation
    g = golden("steps")
    case = sim.RigidSphereCase(nz=64, nr=32, dx=2.0 / 64, r_sphere=0.125, z_cm=0.5)
    s = RigidSphereSimulation(case, device="cuda")
    np.testing.assert_array_equal(s.vorticity.cpu().numpy(), g["rigid/omega0"])
    np.testing.assert_array_equal(s.char_func.cpu().numpy() > 0.5, g["rigid/chi"] > 0.5)
    dts = []
    for n in range(40):
        s.step()
        dts.append(s.dt)
        if n + 1 in (1, 10, 40):
            for f, t in (("omega", s.vorticity), ("psi", s.psi), ("u_z", s.u_z), ("u_r", s.u_r)):
                err = rel_l2(t.cpu().numpy(), g[f"rigid/{f}_{n + 1}"])
                assert err < 1e-12, (f, n + 1, err)
    np.testing.assert_allclose(dts, g["rigid/dt"], rtol=1e-13)


@pytest.mark.parametrize("steps", [20])
def test_rigid_sphere_full_size_against_oracle(steps):
    """512 x 256 (z in [0, 2], r in [0, 1], dx = 1/256, sphere 0.0625 at z = 0.5)."""
    from pyaxisymflow_gb300.simulation import RigidSphereSimulation
    case = sim.RigidSphereCase()
    st, coords = sim.rigid_sphere_init(case, K)
    solver = K.FastDiagonalisationStokesSolver(case.nr, case.nz, case.dx)
    adv = K.gen_advect_vorticity_via_eno3(case.dx, case.nr, case.nz)
    s = RigidSphereSimulation(case, device="cuda")
    for _ in range(steps):
        sim.rigid_sphere_step(case, st, coords, solver, adv, K)
        s.step()
    for f, t, ref in (("omega", s.vorticity, st.vorticity), ("psi", s.psi, st.psi),
                      ("u_z", s.u_z, st.u_z), ("u_r", s.u_r, st.u_r)):
        err = rel_l2(t.cpu().numpy(), ref)
        assert err < 1e-12, (f, err)
    assert abs(s.Cd - st.Cd) <= 1e-10 * abs(st.Cd)


def test_soft_sphere_loop_against_golden(golden):
    """Elasto path end to end: eta advection, level-set pinning, least-squares
    extrapolation, neo-Hookean stress and its curl, tether penalisation."""
    from pyaxisymflow_gb300.simulation import SoftSphereSimulation
    g = golden("soft")
    case = sim.SoftSphereCase(nz=64, nr=32, dx=1.0 / 64, r_ball=0.15, lam=1e6)
    s = SoftSphereSimulation(case, device="cuda")
    s.run(12)
    for f, t in (("omega", s.vorticity), ("eta1", s.eta1), ("eta2", s.eta2),
                 ("phi", s.ball_phi), ("chi", s.ball_char_func)):
        err = rel_l2(t.cpu().numpy(), g[f"soft/{f}_12"])
        assert err < 1e-12, (f, err)
    assert abs(s.t - float(g["soft/t_12"])) <= 1e-13 * float(g["soft/t_12"])


@pytest.mark.parametrize("nr,nz", [(3, 3), (33, 31), (5, 1025)])
def test_sphere_passes_match_the_array_operations(nr, nz):
    """Free stream, maximum speed, penalisation, its vorticity and the drag sum of
    the drop-in loop against the same operations on arrays, with a body over part
    of the grid: the fields and the maximum bit for bit (one rounding per
    operation on both sides), the sum within n unit roundings of its terms."""
    from pyaxisymflow_gb300 import _native as N
    rng = np.random.default_rng(nr * nz)
    uz, ur, w, penal = (rng.standard_normal((nr, nz)) for _ in range(4))
    R = np.repeat((np.arange(nr)[:, None] + 0.5) / nr, nz, 1)
    chi = np.clip(rng.uniform(-2.0, 1.5, (nr, nz)), 0.0, 1.0)
    chi[:, nz // 2:] = 0.0
    lam, dt, dx, add = 1e4, 1e-3, 0.01, 0.25
    dev = {k: torch.tensor(v, device="cuda") for k, v in
           dict(uz=uz, ur=ur, w=w, penal=penal, R=R, chi=chi, oz=0 * uz, orr=0 * ur).items()}
    out = torch.zeros(2, dtype=torch.float64, device="cuda")
    parts = torch.empty(int(N.lib().axi_sphere_penalise_partials(nr, nz)), dtype=torch.float64,
                        device="cuda")
    s = N.stream_of(out)
    N.call("axi_sphere_speed_f64", N.ptr(dev["uz"]), N.ptr(dev["ur"]), add, nr * nz,
           N.ptr(out[:1]), s)
    N.call("axi_sphere_penalise_f64", N.ptr(dev["w"]), N.ptr(dev["penal"]), N.ptr(dev["uz"]),
           N.ptr(dev["ur"]), N.ptr(dev["oz"]), N.ptr(dev["orr"]), N.ptr(dev["chi"]),
           N.ptr(dev["R"]), lam, dt, nr, nz, dx, N.ptr(parts), N.ptr(out[1:]), s)
    uz = uz + add
    umax = (np.abs(uz) + np.abs(ur)).max()
    lc = lam * dt * chi
    pz, pr = (uz + lc * 0.0) / (1 + lc), (ur + lc * 0.0) / (1 + lc)
    dz, dr = pz - uz, pr - ur
    penal[1:-1, 1:-1] = ((dr[1:-1, 2:] - dr[1:-1, :-2]) / (2 * dx)
                         - (dz[2:, 1:-1] - dz[:-2, 1:-1]) / (2 * dx))
    for k, ref in (("uz", pz), ("ur", pr), ("oz", uz), ("orr", ur), ("penal", penal),
                   ("w", w + penal)):
        np.testing.assert_array_equal(dev[k].cpu().numpy(), ref, err_msg=k)
    got = out.cpu().numpy()
    terms = R * chi * pz
    assert got[0] == umax
    assert abs(got[1] - terms.sum()) <= nr * nz * 2.0 ** -52 * np.abs(terms).sum()
    dev["ur"][0, 0] = float("nan")
    N.call("axi_sphere_speed_f64", N.ptr(dev["uz"]), N.ptr(dev["ur"]), add, nr * nz,
           N.ptr(out[:1]), s)
    assert np.isnan(out[0].item())
