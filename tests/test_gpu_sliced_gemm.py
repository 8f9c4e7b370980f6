"""FP64 products on the tensor cores by integer slicing, against long double."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def sliced_gemm(A, B, S=None):
    from pyaxisymflow_gb300 import _native as N
    M, K = A.shape
    Nn = B.shape[0]
    C = torch.empty((M, Nn), dtype=torch.float64, device=A.device)
    work = torch.empty(N.lib().axi_sliced_gemm_work_bytes(M, Nn, K), dtype=torch.uint8,
                       device=A.device)
    N.call("axi_sliced_gemm_f64", N.ptr(C), N.ptr(A), N.ptr(B), N.ptr(S) if S is not None else
           None, M, Nn, K, N.ptr(work), N.stream_of(A))
    return C


def operands(kind, M, N, K):
    rng = np.random.default_rng(M + 3 * N + 7 * K)
    A, B = rng.standard_normal((M, K)), rng.standard_normal((N, K))
    if kind == "graded":        # spread over 30 decades within and across rows
        A *= 10.0 ** rng.uniform(-30, 0, (M, K)) * 10.0 ** rng.uniform(-100, 100, (M, 1))
        B *= 10.0 ** rng.uniform(-30, 0, (N, K)) * 10.0 ** rng.uniform(-100, 100, (N, 1))
    elif kind == "extreme":     # digit sums at their largest: one sign, full digits
        A = np.full((M, K), -(2.0 - 2.0 ** -52))
        B = np.full((N, K), 64.5 / 64 * 1.9999)
        A[:, ::2] = -(1.0 - 2.0 ** -53)
    return A, B


@pytest.mark.parametrize("kind", ["normal", "graded", "extreme"])
@pytest.mark.parametrize("M,N,K", [(128, 32, 16), (1, 1, 1), (128, 32, 80), (129, 33, 17),
                                   (200, 77, 130), (128, 64, 512), (130, 40, 528),
                                   (256, 96, 1040),
                                   # tiles of 128 x 16: up to 38 in four shares of
                                   # K (above), to 76 in two, to 152 whole, else wide
                                   (640, 150, 200), (700, 145, 33), (1024, 200, 300),
                                   (2560, 130, 48), (1290, 290, 528), (1280, 256, 1040)])
def test_sliced_gemm_is_exact_to_the_row_scales(kind, M, N, K):
    A, B = operands(kind, M, N, K)
    C = sliced_gemm(torch.tensor(A).cuda(), torch.tensor(B).cuda()).cpu().numpy()
    # long double products of up to 48 rows (first, last, seeded ones between)
    rows = np.unique(np.concatenate([[0, M - 1], np.random.default_rng(1).integers(0, M, 46)]))
    A, C = A[rows], C[rows]
    ref = A.astype(np.longdouble) @ B.T.astype(np.longdouble)
    # per element of K, in units of the scales' product: the dropped plane
    # products are at most 7 * 2^-62 (and 6 * 2^-70 ...), each operand is off by
    # at most 2^-63, together 8.1 * 2^-62; then one rounding to FP64 (long double
    # may itself be off by K ulps of 2^-64)
    ea = np.ldexp(1.0, np.frexp(np.abs(A).max(axis=1))[1]).astype(np.longdouble)
    eb = np.ldexp(1.0, np.frexp(np.abs(B).max(axis=1))[1]).astype(np.longdouble)
    tol = K * 8.1 * 2.0 ** -62 * ea[:, None] * eb[None, :] + np.abs(ref) * np.longdouble(2.0) ** -52.9
    assert np.all(np.abs(C - ref) <= tol), float(np.max(np.abs(C - ref) / tol))


def test_sliced_gemm_scale_zero_rows_and_values_that_are_not_finite():
    A, B = operands("normal", 140, 50, 100)
    S = np.random.default_rng(2).standard_normal((140, 50))
    A[3] = 0.0
    A[7] *= 5e-320 / np.abs(A[7]).max()      # a subnormal row
    B[5, 9] = np.inf
    B[6, 1] = np.nan
    C = sliced_gemm(*(torch.tensor(x).cuda() for x in (A, B, S))).cpu().numpy()
    ok = np.ones(50, bool)
    ok[[5, 6]] = False
    assert np.all(C[3, ok] == 0.0)
    assert np.all(np.isnan(C[:, ~ok]))
    ref = (A @ B[ok].T) * S[:, ok]
    normal = np.arange(140) != 7
    assert np.allclose(C[normal][:, ok], ref[normal], rtol=1e-12, atol=1e-13)
    # 100 subnormal inputs, each known to half of 2^-1074
    assert np.all(np.abs(C[7, ok] - ref[7]) <= 2.0 ** -1074 * 100 * 10)


def solve_error(solver, ref_solver, w):
    psi = torch.zeros_like(w)
    solver.solve(psi, w)
    ref = np.zeros(w.shape)
    ref_solver.solve(ref, w.cpu().numpy())
    return float(np.linalg.norm(psi.cpu().numpy() - ref) / np.linalg.norm(ref))


@pytest.mark.parametrize("nr,nz", [(8, 9), (31, 33), (64, 128), (129, 257), (200, 600)])
def test_spectral_solve_on_sliced_products(nr, nz):
    from oracle import kernels as OK
    from pyaxisymflow_gb300.kernels.FastDiagonalisationStokesSolver import (
        FastDiagonalisationStokesSolver)
    solver = FastDiagonalisationStokesSolver(nr, nz, 1.0 / nr)
    ref = OK.FastDiagonalisationStokesSolver(nr, nz, 1.0 / nr)
    wide = torch.tensor(np.random.default_rng(nr).standard_normal((nr, nz + 5))).cuda()
    # contiguous, a strided window (odd offset), and in place
    assert solve_error(solver, ref, wide[:, :nz].contiguous()) < 1e-12
    assert solve_error(solver, ref, wide[:, 3:nz + 3]) < 1e-12
    w = wide[:, :nz].contiguous()
    out = torch.zeros_like(w)
    solver.solve(out, w)
    solver.solve(w, w)
    assert torch.equal(out, w)
    assert solver.engine.status() == 0
