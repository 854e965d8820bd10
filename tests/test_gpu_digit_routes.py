"""Calls whose products run on digits at these sizes and on the FP64 kernels in the
smaller problems of the other tests: several columns per SNP, the adjoint, a triangular
operand longer than one launch's K.  Tolerances are those of the same calls there (the
FP64 path against the oracle, 1e-12; the adjoint against the CPU gradient, 1e-9)."""
import ctypes as C
import subprocess

import numpy as np
import pytest

from oracle import fgls_oracle as O
from test_gpu_parity import CHOL_TOL, EIGEN_TOL, check

pytestmark = pytest.mark.gpu


def assert_on_digits(e, run):
    """The call's products wait on the tensor cores' pipelines: a limit of 1 ns ends it."""
    from fgls_gb300 import FGLSError
    from fgls_gb300.engine import ETIMEOUT
    e.set_wait_limit(1)
    with pytest.raises(FGLSError) as ei:
        run()
    assert ei.value.code == ETIMEOUT, ei.value
    e.set_wait_limit(0)


@pytest.mark.parametrize("variant", ["eigen", "chol"])
@pytest.mark.parametrize("wXR,dosages", [(2, False), (3, False), (3, True)])
def test_columns_per_snp(variant, wXR, dosages):
    from fgls_gb300 import Engine, datagen
    t = 2 if variant == "eigen" else 1
    pb = datagen.make_problem(700, 300, t, wXL=3, wXR=wXR, seed=70 + wXR, hsig_uniform=True)  # blocks of 256 and 44
    if dosages:
        rng = np.random.default_rng(71)
        pb.XR = np.clip(pb.XR + 0.2 * rng.standard_normal(pb.XR.shape), 0.0, 2.0)
    with Engine(pb.n, 3, wXR, t, 256, variant=variant) as e:
        e.set_problem(pb.Phi, pb.XL, pb.Y, pb.h, pb.sigma)
        e.select_trait(0)
        B, V = e.run_snps(pb.XR)
        assert_on_digits(e, lambda: e.run_snps(pb.XR))
    Br, Vr = O.fgls_eigen(pb) if variant == "eigen" else O.fgls_chol(pb, 256)
    check(O.compare(B, V, Br, Vr), EIGEN_TOL if variant == "eigen" else CHOL_TOL)


@pytest.mark.parametrize("n,t,m,x_b", [(1000, 5, 600, 256), (1500, 40, 1030, 1024)])  # the second: dY's products too
def test_adjoint(n, t, m, x_b):
    """Other values of h and sigma before, the last block shorter than the others."""
    import torch
    from fgls_gb300 import Engine, datagen
    pb = datagen.make_problem(n, m, t, seed=n, hsig_uniform=True)
    rng = np.random.default_rng(n)
    bbar = rng.standard_normal((t, m, pb.p))
    dX = torch.from_numpy(np.ascontiguousarray(pb.XR.T)).cuda()
    dB = torch.from_numpy(bbar).cuda()
    torch.cuda.synchronize()
    with Engine(n, 3, 1, t, x_b, variant="eigen") as e:
        def gradient():
            e.adjoint_reset()
            for ib in range(0, m, x_b):
                e.adjoint_block_device(dX[ib].data_ptr(), min(x_b, m - ib), dB[0, ib].data_ptr(), m * pb.p)
            return e.adjoint_read()
        e.set_problem(pb.Phi, pb.XL, pb.Y, 1.0 - pb.h, 2.0 * pb.sigma)
        gradient()
        e.set_hsigma(pb.h, pb.sigma)
        dh, ds, dY = gradient()
        ll, dll = e.reml()
        W, Z = e.eigen()
        assert_on_digits(e, gradient)
    rh, _, rY = O.eigen_adjoint(Z, W, pb.XL, pb.Y, pb.h, pb.sigma, pb.XR, bbar)
    assert np.allclose(dh, rh, rtol=1e-9, atol=1e-12 * np.abs(rh).max())
    assert np.abs(ds).max() < 1e-9 * np.abs(dh).max()  # beta is scale-invariant in sigma
    assert np.allclose(dY, rY, rtol=1e-9, atol=1e-9 * np.abs(rY).max())
    rll, rdll = O.reml(Z, W, pb.XL, pb.Y, pb.h, pb.sigma)
    assert np.allclose(ll, rll, rtol=1e-10)
    assert np.allclose(dll, rdll, rtol=1e-9, atol=1e-12)


def test_triangular_operand_longer_than_one_launch():
    """L^-1 X at n = 20600 (160 K-steps a launch: 20480), against the Woodbury form of
    M = s (I + h U U^T), whose products are short."""
    from fgls_gb300 import Engine, datagen
    rng = np.random.default_rng(20)
    n, w, x, h, s = 20600, 3, 200, 0.6, 1.4
    U = rng.standard_normal((n, 5)) / np.sqrt(n)
    Phi = U @ U.T
    Phi = 0.5 * (Phi + Phi.T)
    Phi[np.diag_indices(n)] += 1.0
    XL = rng.standard_normal((n, w))
    XL[:, 0] = 1.0
    XR = datagen.hardcall_genotypes(rng, n, x)
    y = rng.standard_normal(n)
    with Engine(n, w, 1, 1, x, variant="chol") as e:
        e.set_problem(Phi, XL, y[:, None], np.array([h]), np.array([s]))
        e.select_trait(0)
        B, V = e.run_block(XR)
        assert_on_digits(e, lambda: e.run_block(XR))
    # M = s ((h + 1 - h) I + h U U^T); M^-1 = (I - U (I / h + U^T U)^-1 U^T) / s
    core = np.linalg.inv(np.eye(5) / h + U.T @ U)

    def dot(a, b):
        return (a.T @ b - (a.T @ U) @ core @ (U.T @ b)) / s
    null = np.linalg.solve(dot(XL, XL), dot(XL, y))
    r = y - XL @ null
    res = dot(r, r) / (n - w)
    LR, Ry = dot(XL, XR), dot(XR, y)
    RU = XR.T @ U
    RR = ((XR * XR).sum(0) - np.einsum("ka,ab,kb->k", RU, core, RU)) / s
    for k in range(x):
        S = np.block([[dot(XL, XL), LR[:, k:k + 1]], [LR[:, k:k + 1].T, np.array([[RR[k]]])]])
        b = np.linalg.solve(S, np.append(dot(XL, y), Ry[k]))
        se = np.sqrt(np.diag(np.linalg.inv(S)) * res)
        assert np.max(np.abs(B[0, k] - b) / (np.abs(b) + se)) <= 1e-12
        assert np.max(np.abs(V[0, k][range(w + 1), range(w + 1)] - se) / se) <= 1e-12


CHAIN = r"""
#include "fgls_common.cuh"
__global__ void k(const double* x, double* rcp, double* rsq, int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) { rcp[i] = fgls::chain_rcp(x[i]); rsq[i] = fgls::chain_rsqrt(x[i]); }
}
extern "C" int run(const double* x, double* rcp, double* rsq, int n) {
  k<<<(n + 255) / 256, 256>>>(x, rcp, rsq, n);
  return (int)cudaDeviceSynchronize();
}
"""


def test_reciprocals_on_a_short_chain(tmp_path):
    """chain_rcp and chain_rsqrt: half an ulp for the last rounding, and what their series
    leave off, 2^-66 and 2^-63.7 of the result (0.001 ulp); CUDA's own functions
    (at most one ulp) outside of the range that the mantissa moves cover."""
    import torch
    if np.finfo(np.longdouble).nmant < 100:
        pytest.skip("needs a quad longdouble")
    src, so = tmp_path / "chain.cu", tmp_path / "chain.so"
    src.write_text(CHAIN)
    from fgls_gb300 import build as B
    subprocess.run([B.nvcc(), B.ARCH, "-O3", "-std=c++17", "-shared", "-Xcompiler", "-fPIC", "-I", B.INCLUDE, "-I",
                    B.CSRC, "--expt-relaxed-constexpr", str(src), "-o", str(so)], check=True)
    rng = np.random.default_rng(21)
    ex = np.repeat(np.arange(0, 2047, dtype=np.uint64), 200)
    man = rng.integers(0, 1 << 52, ex.size, dtype=np.uint64)
    man[::200], man[1::200], man[2::200] = 0, (1 << 52) - 1, 1 << 29  # the ends, and one bit past the FP32 seed's
    x = ((ex << np.uint64(52)) | man).view(np.float64)
    x = np.concatenate([x, [0.0, -0.0, np.inf, np.nan], -x[::7]])
    d = torch.from_numpy(x).cuda()
    out = torch.empty((2, x.size), dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    lib = C.CDLL(str(so))
    assert lib.run(C.c_void_p(d.data_ptr()), C.c_void_p(out[0].data_ptr()), C.c_void_p(out[1].data_ptr()), x.size) == 0
    rcp, rsq = out.cpu().numpy()
    q = x.astype(np.longdouble)
    with np.errstate(all="ignore"):
        for got, ref, lo, hi in ((rcp, 1 / q, 2, 0x7fc), (rsq, 1 / np.sqrt(q), 1, 0x7fe)):
            r64 = ref.astype(np.float64)
            same = ~np.isfinite(r64)
            assert np.array_equal(np.isnan(got[same]), np.isnan(r64[same]))
            inf = np.isinf(r64)
            assert np.array_equal(got[inf], r64[inf])
            fin = np.isfinite(r64)
            e = (x.view(np.uint64) >> np.uint64(52)).astype(np.int64) & 0x7ff
            ulp = np.abs((got[fin].astype(np.longdouble) - ref[fin]) / np.spacing(np.abs(r64[fin])))
            assert ulp[(e[fin] >= lo) & (e[fin] <= hi)].max() <= 0.51
            assert ulp.max() <= 1.0
