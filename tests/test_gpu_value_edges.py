"""The FP64 kernels' shortcuts (division by a known divisor, comparisons and
widening on the integer pipe, zero regions) against numpy at the edges of what
they take: exponent windows, signed zeros, subnormal numbers, infinities, NaN."""
import numpy as np
import pytest
import torch

from oracle import kernels as K

pytestmark = [pytest.mark.gpu, pytest.mark.filterwarnings("ignore::RuntimeWarning")]


def dev(a):
    return torch.tensor(np.ascontiguousarray(a), device="cuda")


def same(got, want):
    """Equal values and signs; NaN where NaN."""
    got = got.cpu().numpy() if isinstance(got, torch.Tensor) else got
    np.testing.assert_array_equal(got, want)
    ok = ~np.isnan(want)
    np.testing.assert_array_equal(np.signbit(got[ok]), np.signbit(want[ok]))


def values(exponents, rng, n=3):
    """Both signs of random, all-ones and power-of-two significands."""
    m = np.concatenate([[1.0, 2.0 - 2.0 ** -52, 1.0 + 2.0 ** -52], rng.uniform(1, 2, n)])
    v = np.ldexp(m[None, :], np.asarray(exponents)[:, None]).ravel()
    return np.concatenate([v, -v])


SPECIAL = np.array([0.0, -0.0, np.inf, -np.inf, np.nan, 5e-324, -5e-324, 2.2250738585072009e-308,
                    1.7976931348623157e308])


def test_quotients_by_a_known_divisor():
    """The window takes divisors from 2^-400 to 2^400 and dividends from 2^-500 to
    2^500 (biased exponents 623 .. 1423 and 523 .. 1523): correctly rounded in and
    outside it."""
    from pyaxisymflow_gb300 import _native as N
    rng = np.random.default_rng(0)
    dividends = np.concatenate([values([-1074, -1022, -600, -501, -500, -499, -1, 0, 1, 53, 499,
                                        500, 501, 600, 1023], rng), SPECIAL,
                                np.ldexp(rng.uniform(1, 2, 2000), rng.integers(-520, 520, 2000))])
    divisors = np.concatenate([values([-1000, -402, -401, -400, -399, -1, 0, 3, 399, 400, 401,
                                       1000], rng, 2), [np.inf, np.nan, 0.0, -0.0, 1e-310]])
    n = dividends.size
    u_r = np.zeros((3, 4 * n + 4))
    u_r[1, 2:4 * n + 2:4] = dividends          # cell 4 k + 1 sees it minus zero
    u, z, out = dev(u_r), dev(np.zeros_like(u_r)), dev(np.zeros_like(u_r))
    s = N.stream_of(out)
    for d in divisors:
        dx = d * 0.5
        out.zero_()
        N.call("axi_vorticity_from_velocity_unb_f64", N.ptr(out), N.ptr(z), N.ptr(u), 3,
               u_r.shape[1], float(dx), s)
        want = (u_r[1, 2:] - u_r[1, :-2]) / (2 * dx) - 0.0 / (2 * dx)
        same(out[1, 1:-1], want)


def velocities(nr, nz, rng):
    u = rng.standard_normal((2, nr, nz))
    u[:, 3, :] = 0.0
    u[:, 4, ::2] = -0.0
    u[0, 5, 1::2] = -u[0, 5, :-1:2][:nz // 2]   # u0 = -u1 exactly
    u[1, 7, :] = -u[1, 6, :]
    u[:, 9, 5:9] = [np.inf, -np.inf, np.nan, 5e-324]
    u[0, 10, 11:13] = [-5e-324, 5e-324]
    return u


@pytest.mark.parametrize("nr,nz", [(13, 40), (16, 64), (33, 95)])
def test_upwind_choice_and_zero_regions_of_the_advection(nr, nz):
    from pyaxisymflow_gb300.elasto_kernels.advect_refmap_via_eno3 import gen_advect_refmap_via_eno3
    from pyaxisymflow_gb300.kernels.advect_vorticity_via_eno3 import gen_advect_vorticity_via_eno3
    rng = np.random.default_rng(nz)
    dx, dt = 1.0 / nz, 0.3 / nz
    uz, ur = velocities(nr, nz, rng)
    w = rng.standard_normal((nr, nz))
    w[8, 3:6] = [0.0, -0.0, np.nan]
    # reference maps that are zero but for one block; -0 and infinities beside it
    e1, e2 = np.zeros((nr, nz)), np.zeros((nr, nz))
    e1[2:5, 30:34], e2[2:5, 30:34] = rng.standard_normal((2, 3, 4))
    e1[6, 20:23], e2[0, 10] = [-0.0, 1e-320, np.inf], -0.0
    for fields, ref_fn, fn in (
            ([w], K.gen_advect_vorticity_via_eno3(dx, nr, nz),
             gen_advect_vorticity_via_eno3(dx, nr, nz)),
            ([e1, e2], K.gen_advect_refmap_via_eno3(dx, nr, nz),
             gen_advect_refmap_via_eno3(dx, nr, nz))):
        ref, got = [f.copy() for f in fields], [dev(f) for f in fields]
        ref_fn(*ref, uz, ur, dt)
        fn(*got, dev(uz), dev(ur), dt)
        for g, r in zip(got, ref):
            same(g, r)


@pytest.mark.parametrize("w", [0.1, 1e-300, 5e-320, 1e300])
def test_heaviside_at_the_ends_of_its_band(w):
    from pyaxisymflow_gb300.kernels.smooth_Heaviside import smooth_Heaviside
    up, down = np.nextafter(w, np.inf), np.nextafter(w, 0)
    phi = np.concatenate([s * np.array([w, up, down, 0.5 * w, 0.0, 2 * w, 1e-320, 1.0])
                          for s in (1, -1)] + [SPECIAL, [1e305, -1e305]])
    old = np.array([0.0, -0.0, 1.0, -3.0, 1e-310, np.inf, np.nan])
    P, H = (np.ascontiguousarray(a) for a in np.meshgrid(phi, old))
    ref, got = H.copy(), dev(H)
    K.smooth_Heaviside(ref, P, w)
    smooth_Heaviside(got, dev(P), w)
    got = got.cpu().numpy()
    band = np.abs(P) < w                       # sin of CUDA and of numpy: 2 ulp of the bracket
    same(got[~band], ref[~band])
    np.testing.assert_allclose(got[band], ref[band], rtol=4e-16, atol=4e-16)


def test_widening_of_floats():
    from pyaxisymflow_gb300 import _native as N
    e = np.arange(256, dtype=np.uint32)[:, None] << 23
    m = np.array([0, 1, 2, 0x400000, 0x7ffffe, 0x7fffff, 0x2aaaaa], dtype=np.uint32)
    bits = (e | m).ravel()
    x = np.concatenate([bits, bits | np.uint32(1 << 31)]).view(np.float32)
    y, f = torch.empty(x.size, dtype=torch.float64, device="cuda"), dev(x)
    N.call("axi_widen_f32_to_f64", N.ptr(y), N.ptr(f), x.size, N.stream_of(y))
    same(y, x.astype(np.float64))
    add = np.random.default_rng(1).standard_normal(x.size)
    for name, want in (("axi_add_f32_to_f64", add + x.astype(np.float64)),):
        t = dev(add)
        N.call(name, N.ptr(t), N.ptr(f), x.size, N.stream_of(t))
        same(t, want)
    out, t = torch.empty_like(y), dev(add)
    N.call("axi_sum_f32_to_f64", N.ptr(out), N.ptr(t), N.ptr(f), x.size, N.stream_of(t))
    same(out, add + x.astype(np.float64))
    same(t, add)


def extrapolate(mod, phi, eta, zone, nr, nz, z):
    conv = dev if mod is not K else (lambda a: a)
    inside = conv(phi > 0)
    e = [conv(x.copy()) for x in eta]
    d = [conv(np.zeros((2 * nr, nz))) for _ in range(3)]
    try:
        mod.extrapolate_eta_with_least_squares(inside, conv(phi), *e, *d, zone, nr, conv(z))
        failed = None
    except (ValueError, RuntimeError) as x:
        failed = str(x)
    return e, failed


@pytest.mark.parametrize("cells", [3, 8, 9, 14])
def test_extrapolation_within_and_beyond_its_counted_sweeps(cells):
    """Eight sweeps are issued one launch each; bands that need more go on in the
    finishing pass."""
    from pyaxisymflow_gb300.elasto_kernels import extrapolate_eta_using_least_squares_unb as G
    nr, nz = 32, 64
    dx = 1.0 / nz
    z = (np.arange(nz) + 0.5) * dx
    Z, R = np.meshgrid(z, z[:nr])
    phi = 0.14 - np.sqrt((Z - 0.5) ** 2 + R ** 2)
    eta = [Z + 0.05 * np.sin(7 * R), R * (1 + 0.1 * np.cos(5 * Z))]
    ref, failed = extrapolate(K, phi, eta, cells * dx, nr, nz, z)
    assert failed is None
    got, failed = extrapolate(G, phi, eta, cells * dx, nr, nz, z)
    assert failed is None
    for g, r in zip(got, ref):
        same(g, r)


def test_extrapolation_window_that_leaves_the_grid():
    """A front cell of the first column whose one known neighbour lies straight
    below: its window starts left of the grid. The maps stay as they were."""
    from pyaxisymflow_gb300.elasto_kernels import extrapolate_eta_using_least_squares_unb as G
    nr, nz = 16, 32
    dx = 1.0 / nz
    z = (np.arange(nz) + 0.5) * dx
    phi = np.full((nr, nz), -1.5 * dx)
    phi[5:8, 0] = 0.5 * dx
    eta = list(np.random.default_rng(0).standard_normal((2, nr, nz)))
    assert "grid" in extrapolate(K, phi, eta, 2 * dx, nr, nz, z)[1]
    got, failed = extrapolate(G, phi, eta, 2 * dx, nr, nz, z)
    assert failed is not None
    for g, e in zip(got, eta):
        same(g, e)
