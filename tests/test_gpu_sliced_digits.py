"""The sliced FP64 product bit for bit: the sum of the digit products that the
method keeps, formed in integers on the host and rounded once, also where the
accumulators come closest to the 2^24 up to which FP32 holds every integer."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

DIGITS = 8


def value(digits, scale_exp):
    """Doubles sum_i d_i 2^(-6 - 8 i) 2^scale_exp (exact: at most 53 bits)."""
    q = sum(int(1) * digits[..., i].astype(object) * 256 ** (7 - i) for i in range(DIGITS))
    x = np.array([float(v) for v in q.ravel()]).reshape(q.shape)
    assert all(int(a) == b for a, b in zip(x.ravel(), q.ravel()))
    return np.ldexp(x, scale_exp - 62)


def digits_of(x):
    """The eight digits of each element below its row's power of two, the last one
    rounded to nearest (halves away from zero)."""
    e = np.frexp(np.abs(x).max(axis=1))[1]
    y = np.ldexp(x.astype(np.longdouble), (62 - e)[:, None])
    q = (np.sign(y) * np.floor(np.abs(y) + 0.5)).astype(np.int64)
    u = q.view(np.uint64) + np.uint64(0x8080808080808080)
    d = np.stack([((u >> np.uint64(56 - 8 * i)) & np.uint64(255)).astype(np.int64) - 128
                  for i in range(DIGITS)], axis=-1)
    return d, e


def host_product(A, B):
    """The kept digit products, exactly, rounded once; and the largest group sum
    that a run of 128 K elements forms."""
    (a, ea), (b, eb) = digits_of(A), digits_of(B)
    total = np.zeros((A.shape[0], B.shape[0]), dtype=object)
    largest = 0
    for d in range(DIGITS):
        group = 0
        for k0 in range(0, A.shape[1], 128):
            s = sum(a[:, k0:k0 + 128, i] @ b[:, k0:k0 + 128, d - i].T for i in range(d + 1))
            largest = max(largest, int(np.abs(s).max()))
            group = group + s
        total += group.astype(object) * 256 ** (7 - d)
    out = np.empty(total.shape)
    for (m, n), t in np.ndenumerate(total):
        out[m, n] = np.ldexp(float(t), int(ea[m] + eb[n]) - 68)   # an int rounds to even
    return out, largest


def largest_operands(M, N, K, rng):
    """One sign, digits at or next to -128 in as many places as 53 bits allow, the
    left operand led by -32 (the largest that keeps six full digits below), the
    right one's scale set by an element outside the first 128."""
    def near(shape):
        d = np.zeros(shape + (DIGITS,), dtype=np.int64)
        d[..., 1:7] = rng.integers(-128, -119, shape + (6,))
        return d
    a = near((M, K))
    a[..., 0], a[..., 6] = -32, -128
    b = near((N, K))
    b[..., 1], b[..., 7] = -128, -128
    b[:, 128:, 0] = -32
    b[:, 128:, 6:] = (-128, 0)
    return value(a, 3), value(b, -2)


def gpu_product(A, B):
    from pyaxisymflow_gb300 import _native as N
    a, b = torch.tensor(A).cuda(), torch.tensor(B).cuda()
    (M, K), n = A.shape, B.shape[0]
    out = torch.empty((M, n), dtype=torch.float64, device="cuda")
    work = torch.empty(N.lib().axi_sliced_gemm_work_bytes(M, n, K), dtype=torch.uint8,
                       device="cuda")
    N.call("axi_sliced_gemm_f64", N.ptr(out), N.ptr(a), N.ptr(b), None, M, n, K, N.ptr(work),
           N.stream_of(a))
    return out.cpu().numpy()


# tiles of 16 columns (up to 152 of them) and of 32
@pytest.mark.parametrize("M,N", [(64, 24), (256, 1300)])
@pytest.mark.parametrize("K", [129, 1153])
def test_accumulators_near_their_limit(M, N, K):
    rng = np.random.default_rng(K)
    rows, cols = min(M, 24), min(N, 24)
    A, B = largest_operands(rows, cols, K, rng)
    ref, largest = host_product(A, B)
    # 32 * 128 + 6 * 124^2 on average per element of K, of at most 2^14 * 8
    assert 0.70 * 2 ** 24 < largest < 2 ** 24
    reps = (-(-M // rows), 1), (-(-N // cols), 1)
    C = gpu_product(np.tile(A, reps[0])[:M], np.tile(B, reps[1])[:N])
    np.testing.assert_array_equal(C, np.tile(ref, (reps[0][0], reps[1][0]))[:M, :N])


@pytest.mark.parametrize("M,N,K", [(40, 33, 17), (130, 20, 300)])
def test_digits_of_both_signs(M, N, K):
    rng = np.random.default_rng(M)
    A = rng.standard_normal((M, K)) * 10.0 ** rng.uniform(-8, 0, (M, K))
    B = rng.standard_normal((N, K)) * 10.0 ** rng.uniform(-8, 0, (N, K))
    np.testing.assert_array_equal(gpu_product(A, B), host_product(A, B)[0])
