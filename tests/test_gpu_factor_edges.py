"""The factorizations and small products at the edges of their blocks: 64-column
Cholesky blocks, 512-column panels, inverse merges, 64-column tridiagonalization
panels, 64-row leaves, 512-reflector back-transform blocks, 32 x 8 and 64 x 64
tiles, four-trait REML groups.

Bounds.  FP64 products: K terms, 2^-53 each, of sum |a||b|.  Eigenpairs: backward
stable steps, 40 n 2^-53 of the largest eigenvalue for residuals and eigenvalues
and 40 n 2^-53 for orthogonality.  Chol effects: the gate of the FP64 path against
the oracle (1e-12).  REML: the roots' agreement with the oracle's fit (1e-8), as in
test_gpu_reml.py.
"""
import numpy as np
import pytest

from oracle import fgls_oracle as O
from test_gpu_digit_gemm import product

pytestmark = pytest.mark.gpu
EPS = 2.0 ** -53


@pytest.mark.parametrize("M,N,K", [(1, 1, 1), (31, 7, 31), (33, 9, 33), (64, 64, 64), (65, 3, 200), (800, 800, 70)])
@pytest.mark.parametrize("tA", [0, 1])
@pytest.mark.parametrize("tB", [0, 1])
def test_fp64_product(M, N, K, tA, tB):
    rng = np.random.default_rng(M + N + K)
    A, B, C0 = rng.standard_normal((M, K)), rng.standard_normal((K, N)), rng.standard_normal((M, N))
    out = product(A, B, C0, tA, tB, -0.5, 2.0, digits=0)
    tol = 2 * (K + 3) * EPS * (0.5 * np.abs(A) @ np.abs(B) + 2 * np.abs(C0))
    assert (np.abs(out - (2.0 * C0 - 0.5 * (A @ B))) <= tol).all()


@pytest.mark.parametrize("n", [63, 64, 65, 127, 129, 511, 512, 513, 577, 1025, 1100])
@pytest.mark.parametrize("precision", ["fp64", "split"])
def test_chol_at_block_edges(n, precision):
    from fgls_gb300 import Engine, datagen
    m = 40
    pb = datagen.make_problem(n, m, 1, wXL=2, seed=n, hsig_uniform=True)
    with Engine(n, pb.wXL, 1, 1, m, variant="chol", precision=precision, slices=9) as e:
        e.set_problem(pb.Phi, pb.XL, pb.Y, pb.h, pb.sigma)
        e.select_trait(0)
        B, V = e.run_snps(pb.XR)
    Br, Vr = O.fgls_chol(pb, m)
    d = O.compare(B, V, Br, Vr)
    gate = 1e-12 if precision == "fp64" else 1e-10
    assert d["finite"] and d["beta_se_scaled"] < gate and d["se_rel"] < gate and d["upper_abs_max"] == 0.0, d


def matrix(kind, n, rng):
    if kind == "diagonal":
        return np.diag(rng.uniform(1.0, 2.0, n))
    if kind == "few":  # three eigenvalues: everything deflates, with rotations
        Q, _ = np.linalg.qr(rng.standard_normal((n, n)))
        return (Q * rng.choice([1.0, 2.0, 5.0], n)) @ Q.T
    G = rng.standard_normal((n, 2 * n))
    return G @ G.T / (2 * n) * (1e7 if kind == "large" else 1.0)


@pytest.mark.parametrize("n", [2, 3, 4, 63, 64, 65, 66, 67, 128, 130, 515, 580])
@pytest.mark.parametrize("kind", ["kinship", "large", "few", "diagonal"])
def test_eigendecomposition_at_panel_edges(n, kind):
    from fgls_gb300 import Engine
    rng = np.random.default_rng(n)
    P = matrix(kind, n, rng)
    P = np.tril(P) + np.tril(P, -1).T
    with Engine(n, 1, 1, 1, 4, variant="eigen") as e:
        e.set_problem(P, np.ones((n, 1)), rng.standard_normal((n, 1)), np.array([0.5]), np.ones(1))
        W, Z = e.eigen()
    top = np.abs(W).max()
    tol = 40 * n * EPS
    assert (np.diff(W) >= 0).all()
    assert np.abs(P @ Z - Z * W).max() <= tol * top
    assert np.abs(Z.T @ Z - np.eye(n)).max() <= tol
    assert np.abs(W - np.linalg.eigvalsh(P)).max() <= tol * top


@pytest.mark.parametrize("n,t,grid,wXL", [(40, 1, 2, 1), (257, 3, 5, 2), (300, 4, 64, 7), (301, 5, 256, 3)])
def test_reml_groups_and_grids(n, t, grid, wXL):
    from fgls_gb300 import Engine, datagen
    pb = datagen.make_problem(n, 4, t, wXL=wXL, seed=t, hsig_uniform=True, markers=2 * n)
    with Engine(n, wXL, 1, t, 4, variant="eigen") as e:
        e.set_problem(pb.Phi, pb.XL, pb.Y, pb.h, pb.sigma)
        h, sg, ll, dll = e.reml_fit(0.0, 0.99, grid)
        W, Z = e.eigen()
        for j in range(t):
            # every point of the grid and the ends of [0, 0.99] is at most the fit's value
            e.set_hsigma(np.full(t, h[j]), np.full(t, sg[j]))
            e.adjoint_reset()
            at, _ = e.reml()
            assert abs(at[j] - ll[j]) <= 1e-10 * max(1.0, abs(ll[j]))
        x, y = Z.T @ pb.XL, Z.T @ pb.Y
    for j in range(t):
        def value(hh):
            d = 1 / (1 + hh * (W - 1))
            G = x.T @ (d[:, None] * x)
            r = y[:, j] - x @ np.linalg.solve(G, x.T @ (d * y[:, j]))
            s = (d * r * r).sum() / (n - wXL)
            return -0.5 * ((n - wXL) * np.log(s) - np.log(d).sum() + np.linalg.slogdet(G)[1] + (n - wXL))
        best = max(value(0.99 * k / (grid - 1)) for k in range(grid))
        assert ll[j] >= best - 1e-9 * max(1.0, abs(best))
        assert abs(value(h[j]) - ll[j]) <= 1e-10 * max(1.0, abs(ll[j]))
