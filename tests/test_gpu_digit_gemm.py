"""FP64 products through exact sums of FP8 digit products (csrc/fgls_digit_gemm.cu)
at the edges of its tiles, K-steps, accumulator chunks and K splits, against
exactly rounded sums of the entries.

Bound of one entry, with a = 2^ex of the row (at most 4 max|row|), b likewise:
each operand is rounded to 2^-60 of its scale (a b 2^-61 for both) and the
digit pairs beyond level 13 are dropped (11 pairs of 2^8 at 32^-14 and less:
2^-58.5), so K a b 2^-58 in all; one rounding of the result, of alpha and of
beta, and one per K split (at most 76): 80 * 2^-53 of sum|a||b| + |beta C|.
"""
import ctypes as C
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CASES = [  # M, N, K, transA, transB, alpha, beta
    (1, 1, 1, 0, 0, 1.0, 0.0),          # one element
    (128, 256, 128, 1, 0, 1.0, 0.0),    # one K-step, half a pair's rows
    (129, 257, 129, 0, 1, -1.0, 1.0),   # one past the tile on every side
    (255, 31, 1024, 0, 0, 0.5, -2.0),   # largest K of the warp-per-row cut
    (33, 513, 1025, 1, 1, 1.0, 1.0),    # smallest K of the CTA-per-row cut
    (300, 200, 5377, 1, 0, 1.0, 0.0),   # one K-step past an accumulator's exact range
    (260, 40, 20481, 1, 0, -1.0, 1.0),  # one element past a launch's K
    (2600, 2100, 300, 0, 1, 1.0, 0.0),  # more tiles than CTA pairs
]


def two_prod(a, b):
    p = a * b
    ah = a * 134217729.0
    ah = ah - (ah - a)
    al = a - ah
    bh = b * 134217729.0
    bh = bh - (bh - b)
    bl = b - bh
    return p, ((ah * bh - p) + ah * bl + al * bh) + al * bl


def product(A, B, C0, tA, tB, alpha, beta, digits=1):
    """alpha op(A) op(B) + beta C0 of numpy operands in natural orientation."""
    import torch
    from fgls_gb300 import lib

    def dev(x):
        return torch.from_numpy(np.ascontiguousarray(x)).cuda()
    a = dev(A if tA else A.T)  # column-major op(A)^T or A
    b = dev(B if tB else B.T)
    c = dev(C0.T)
    M, K = A.shape
    N = B.shape[1]
    torch.cuda.synchronize()
    rc = lib().fglsgpu_selftest_dgemm(tA, tB, M, N, K, alpha, C.c_void_p(a.data_ptr()), K if tA else M,
                                      C.c_void_p(b.data_ptr()), N if tB else K, beta, C.c_void_p(c.data_ptr()), M,
                                      digits, None)
    assert rc == 0
    return c.cpu().numpy().T


def scale(x, axis):  # 2^ex of each row: the smallest power of two above 2 max
    m = np.abs(x).max(axis=axis)
    return np.where(m > 0, 2.0 ** (np.floor(np.log2(np.where(m > 0, m, 1.0))) + 2), 0.0)


@pytest.mark.parametrize("M,N,K,tA,tB,alpha,beta", CASES)
@pytest.mark.parametrize("kind", ["normal", "calls", "spread"])
def test_digit_product(M, N, K, tA, tB, alpha, beta, kind):
    rng = np.random.default_rng(M * 7 + N * 3 + K)
    A = rng.standard_normal((M, K))
    B = rng.standard_normal((K, N))
    if kind == "calls":
        B = rng.integers(0, 3, size=(K, N)).astype(np.float64)
    if kind == "spread":
        A *= np.exp(3 * rng.standard_normal((M, K)))
        B[:, N // 2] = 0.0
        A[M // 2] *= 1e-200
    C0 = rng.standard_normal((M, N))
    out = product(A, B, C0, tA, tB, alpha, beta)
    sa, sb = scale(A, 1), scale(B, 0)
    where = {(0, 0), (M - 1, N - 1), (M // 2, N // 2), (min(M - 1, 255), min(N - 1, 256))}
    where |= {(int(rng.integers(M)), int(rng.integers(N))) for _ in range(40)}
    for i, j in where:
        p, e = two_prod(A[i], B[:, j])
        ref = math.fsum([alpha * math.fsum(np.concatenate([p, e])), beta * C0[i, j]])
        tol = abs(alpha) * K * sa[i] * sb[j] * 2.0 ** -58
        tol += 80 * 2.0 ** -53 * (abs(alpha) * np.abs(p).sum() + abs(beta * C0[i, j]))
        assert abs(out[i, j] - ref) <= tol, (i, j, out[i, j], ref, tol)


def test_hard_calls_are_exact():
    """Integers below 2^53 throughout: every level is exact, so is the sum."""
    rng = np.random.default_rng(3)
    A = rng.integers(-2 ** 40, 2 ** 40, size=(300, 700)).astype(np.float64)
    B = rng.integers(0, 3, size=(700, 270)).astype(np.float64)
    out = product(A, B, np.zeros((300, 270)), 1, 0, 1.0, 0.0)
    assert np.array_equal(out, A @ B)


def test_nan_and_infinity_stay_in_their_rows_and_columns():
    rng = np.random.default_rng(4)
    A = rng.standard_normal((300, 400))
    B = rng.standard_normal((400, 260))
    A[7, 3] = np.nan
    B[5, 200] = np.inf
    clean = product(np.nan_to_num(A, nan=0.0), np.where(np.isinf(B), 0.0, B), np.zeros((300, 260)), 1, 0, 1.0, 0.0)
    out = product(A, B, np.zeros((300, 260)), 1, 0, 1.0, 0.0)
    bad = np.zeros((300, 260), bool)
    bad[7] = True
    bad[:, 200] = True
    assert not np.isfinite(out[bad]).any()
    assert np.array_equal(out[~bad], clean[~bad])
