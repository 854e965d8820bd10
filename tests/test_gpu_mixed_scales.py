"""FP64 path on inputs whose individuals differ in scale by many orders of magnitude,
against quad arithmetic (numpy longdouble, where it is quad)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

Q = np.longdouble


def gls(Phi, XL, y, h, s, XR):
    """beta (k, wXL + 1) of every column of XR, wXR = 1, in longdouble."""
    n, w = XL.shape
    M = Q(h * s) * Phi.astype(Q)
    M[np.diag_indices(n)] += Q(1 - h) * Q(s)
    L = np.zeros_like(M)
    for j in range(n):
        c = M[j:, j] - L[j:, :j] @ L[j, :j]
        L[j:, j] = c / np.sqrt(c[0])
    T = np.concatenate([XL, y[:, None], XR], 1).astype(Q)
    for i in range(n):
        T[i] = (T[i] - L[i, :i] @ T[:i]) / L[i, i]
    out = np.zeros((XR.shape[1], w + 1), Q)
    for k in range(XR.shape[1]):
        A = np.concatenate([T[:, :w], T[:, w + 1 + k:w + 2 + k]], 1)
        S = np.concatenate([A.T @ A, (A.T @ T[:, w])[:, None]], 1)
        for i in range(w + 1):
            S[i] = S[i] / S[i, i]
            for j in range(w + 1):
                if j != i:
                    S[j] = S[j] - S[j, i] * S[i]
        out[k] = S[:, -1]
    return out


@pytest.mark.parametrize("decades", [0.0, 2.3, 2.5, 6.0])  # of the standard deviations; the rule's line lies at 2.4
def test_chol_with_variances_of_many_sizes(decades):
    """M = D M' D, h = 1, and XL, XR scaled by D (blocks of 256 SNPs run on digits at
    n = 600).  1e-12 of beta on its standard error's scale, the FP64 path's bound."""
    if np.finfo(Q).nmant < 100:
        pytest.skip("needs a quad longdouble")
    from fgls_gb300 import Engine, datagen
    rng = np.random.default_rng(17)
    n, w, k = 600, 3, 12
    Phi, G = datagen.kinship(rng, n, 3000)
    D = 10.0 ** rng.uniform(-decades / 2, decades / 2, n)
    D[:2] = 10.0 ** (-decades / 2), 10.0 ** (decades / 2)
    Phi = Phi * D[:, None] * D
    XL = rng.standard_normal((n, w))
    XL[:, 0] = 1.0
    XL *= D[:, None]
    XR = datagen.hardcall_genotypes(rng, n, 256) * D[:, None]
    y = D * (G @ rng.standard_normal(3000) / np.sqrt(3000))
    ref = gls(Phi, XL, y, 1.0, 1.3, XR[:, :k])
    with Engine(n, w, 1, 1, 256, variant="chol") as e:
        e.set_problem(Phi, XL, y[:, None], np.array([1.0]), np.array([1.3]))
        e.select_trait(0)
        B, V = e.run_block(XR)
    i = np.arange(w + 1)
    err = np.abs((B[0, :k].astype(Q) - ref).astype(float))
    assert np.max(err / (np.abs(ref.astype(float)) + np.abs(V[0, :k, i, i]).T)) <= 1e-12


def test_digit_products_of_mixed_rows():
    """The documented bound of one digit product, K 2^-58 of the row scales, holds for rows
    of mixed magnitude, and is all that holds there: an element 2^-70 of its row's largest
    is lost, which an FP64 product (relative to sum |a||b|) keeps."""
    from test_gpu_digit_gemm import product, scale
    rng = np.random.default_rng(18)
    M, N, K = 130, 40, 256
    A = rng.standard_normal((M, K)) * 2.0 ** rng.integers(-40, 1, (M, K))
    B = rng.standard_normal((K, N)) * 2.0 ** rng.integers(0, 41, (K, N))
    A[0], B[:, 0] = 0.0, 0.0
    A[0, :2] = 2.0 ** 70, 1.0
    B[1, 0] = 1.0
    ref = np.array([[float(np.sum(A[i].astype(np.longdouble) * B[:, j])) for j in range(N)] for i in range(M)])
    mag = np.abs(A) @ np.abs(B)
    for digits, bound in ((1, K * 2.0 ** -58 * np.outer(scale(A, 1), scale(B, 0))), (0, K * 2.0 ** -53 * mag)):
        out = product(A, B, np.zeros((M, N)), 1, 0, 1.0, 0.0, digits)
        assert np.all(np.abs(out - ref) <= bound + 2.0 ** -52 * mag)
        assert out[0, 0] == (0.0 if digits else 1.0)
