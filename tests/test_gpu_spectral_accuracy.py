"""The FP64 spectral solves element by element, against long double on the same
bases, beside the FP64 FMA products of axi_fd_transform_f64."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

EPS = 2.0 ** -53


def fields(nr, nz, dx):
    rng = np.random.default_rng(nr + nz)
    H, L = nr * dx, nz * dx
    R, Z = np.meshgrid((np.arange(nr) + 0.5) * dx, (np.arange(nz) + 0.5) * dx, indexing="ij")
    return {
        "smooth": R * np.exp(-((R / (0.1 * H)) ** 2 + ((Z - L / 2) / (L / 4)) ** 2)),
        "ring": np.exp(-(((R - 0.5 * H) / (0.06 * H)) ** 2 + ((Z - L / 2) / (L / 5)) ** 2)),
        "white": rng.standard_normal((nr, nz)),
        "axis": np.where(R < 4 * dx, rng.standard_normal((nr, nz)), 0.0),
        "mode": R * np.cos(np.pi * Z / L),
    }


def long_double_solve(host, w, rounded=False):
    """The four products in long double; `rounded`: each of them rounded once to
    double, the least that any form with FP64 intermediates does."""
    h = {k: np.asarray(v, dtype=np.longdouble) for k, v in host.items()}

    def store(x):
        return x.astype(np.float64).astype(np.longdouble) if rounded else x

    x = store(w.astype(np.longdouble) @ h["EzinvT"])
    x = store(store(h["Er_inv_w"] @ x) * h["inv_eig"])
    return store(h["Er"] @ store(x @ h["EzT"]))


def fma_solve(eng, w):
    from pyaxisymflow_gb300 import _native as N
    nr, nz = w.shape
    out, work = torch.empty_like(w), torch.empty(2 * nr * nz, dtype=w.dtype, device=w.device)
    d = eng.dev
    N.call("axi_fd_transform_f64", N.ptr(out), nz, N.ptr(w), nz, N.ptr(d["Er_inv_w"]),
           N.ptr(d["EzinvT"]), N.ptr(d["inv_eig"]), N.ptr(d["Er"]), N.ptr(d["EzT"]),
           N.ptr(work), nr, nz, N.stream_of(w))
    return out


def axial_velocity(psi, dx):
    u = np.empty_like(psi)
    u[1:-1] = psi[2:] - psi[:-2]
    u[0] = -psi[2] + 4 * psi[1] - 3 * psi[0]
    u[-1] = psi[-3] - 4 * psi[-2] + 3 * psi[-1]
    return u / (2 * dx * dx * (np.arange(psi.shape[0]) + 0.5))[:, None]


def rows(e, ref):
    """L2 error of every row relative to that row."""
    size = np.sqrt((ref * ref).sum(axis=1))
    return (np.sqrt((e * e).sum(axis=1)) / np.where(size > 0, size, 1)).astype(np.float64)


def solver(kind, nr, nz, dx):
    from pyaxisymflow_gb300.kernels import FastDiagonalisationStokesSolver as S
    from pyaxisymflow_gb300.kernels.FastDiagonalisationPotentialSolver import (
        FastDiagonalisationPotentialSolver)
    from pyaxisymflow_gb300.kernels.implicit_diffusion_solver import ImplicitEulerDiffusionStepper
    return {
        "stokes": lambda: S.FastDiagonalisationStokesSolver(nr, nz, dx),
        "periodic": lambda: S.FastDiagonalisationStokesSolver(
            nr, nz, dx, bc_type=S.NEUMANN_R_PERIODIC_Z),
        "dirichlet": lambda: S.FastDiagonalisationStokesSolver(
            nr, nz, dx, bc_type=S.DIRICHLET_R_PERIODIC_Z),
        "potential": lambda: FastDiagonalisationPotentialSolver(nr, nz, dx),
        "diffusion": lambda: ImplicitEulerDiffusionStepper(1e-2, 1.0, nr, nz, dx),
    }[kind]().engine


@pytest.mark.parametrize("kind,nr,nz", [("stokes", 65, 200), ("stokes", 512, 40),
                                        ("stokes", 1024, 24), ("periodic", 300, 33),
                                        ("dirichlet", 300, 40), ("potential", 130, 48),
                                        ("diffusion", 200, 40)])
def test_rows_next_to_the_axis_are_as_accurate_as_with_fma(kind, nr, nz):
    """At most twice the error of the FMA products (they differ by that much with
    the order of their sums), or of exact products that are each rounded once to
    FP64 (in some rows the FMA sums happen to undo that rounding). With Dirichlet
    rows one nearly singular mode carries a single rounding of either form into
    every row: eight times."""
    dx = 1.0 / nr
    times = 8 if kind == "dirichlet" else 2
    eng = solver(kind, nr, nz, dx)
    for name, w in fields(nr, nz, dx).items():
        wd = torch.tensor(w, device="cuda")
        got = torch.zeros_like(wd)
        eng.transform(got, wd)
        ref = long_double_solve(eng.host, w)
        e, f = (x.cpu().numpy() - ref for x in (got, fma_solve(eng, wd)))
        g = long_double_solve(eng.host, w, rounded=True) - ref
        re, rf, rg = rows(e, ref), rows(f, ref), rows(g, ref)
        bound = np.maximum(np.maximum(times * rf, 2 * rg), 2 * EPS)
        worst = int(np.argmax(re / bound))
        assert np.all(re <= bound), (name, worst, re[worst], rf[worst], rg[worst])
        if kind in ("stokes", "periodic"):
            ue, uf, ug = (np.abs(axial_velocity(x, dx)).max() for x in (e, f, g))
            assert ue <= 2 * max(uf, ug), (name, ue, uf, ug)


@pytest.mark.parametrize("nr,nz", [(8, 9), (33, 40), (200, 77)])
def test_balanced_products_of_any_size_zeros_and_tiny_values(nr, nz):
    """Powers of two of the field change no bit; zero rows, zero fields, a field
    that is subnormal and rows 600 orders of magnitude apart give what the FMA
    products give."""
    dx = 1.0 / nr
    eng = solver("stokes", nr, nz, dx)
    w = np.random.default_rng(nz).standard_normal((nr, nz))
    w[3:5] = 0.0

    def run(x):
        d = torch.tensor(x, device="cuda")
        out = torch.full_like(d, 7.0)
        eng.transform(out, d)
        return out.cpu().numpy(), fma_solve(eng, d).cpu().numpy()

    base, _ = run(w)
    for p in (-900, 900):
        got, _ = run(np.ldexp(w, p))
        np.testing.assert_array_equal(got, np.ldexp(base, p))
    assert not run(0 * w)[0].any()
    got, want = run(np.ldexp(w, -1066))
    # every term and every partial sum of either form off by at most 2^-1074
    h = {k: np.abs(v) for k, v in eng.host.items()}
    err = float(nz + 1)
    err = ((h["Er_inv_w"].sum(axis=1) * err + nr + 1)[:, None] * h["inv_eig"] + 1).max()
    err = h["EzT"].sum(axis=0).max() * err + nz + 1
    err = h["Er"].sum(axis=1).max() * err + nr + 1
    assert np.abs(got - want).max() <= 2 * err * 2.0 ** -1074
    spread = np.ldexp(w, np.linspace(-990, 990, nr).astype(int)[:, None])
    got, want = run(spread)
    assert np.abs(got - want).max() <= 1e-11 * np.abs(want).max()


def test_values_that_are_not_finite_reach_every_cell():
    eng = solver("stokes", 40, 36, 0.02)
    for bad in (np.nan, np.inf, -np.inf):
        w = torch.ones((40, 36), dtype=torch.float64, device="cuda")
        w[5, 7] = bad
        out = torch.zeros_like(w)
        eng.transform(out, w)
        assert not torch.isfinite(out).any()
    w.fill_(1.0)
    eng.transform(out, w)
    assert torch.isfinite(out).all()
