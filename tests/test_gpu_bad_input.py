"""Inputs that no eigendecomposition exists for are refused, and the engine stays usable."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [200, 1100])  # one merge level and several; products on FP64 kernels, on digits
@pytest.mark.parametrize("value", [np.nan, np.inf])
def test_kinship_that_is_not_finite(n, value):
    from fgls_gb300 import Engine, FGLSError, datagen
    pb = datagen.make_problem(n, 40, 2, seed=n, hsig_uniform=True)
    bad = pb.Phi.copy()
    bad[n - 3, n // 3] = bad[n // 3, n - 3] = value
    with Engine(n, 3, 1, 2, 64, variant="eigen") as e:
        e.set_problem(pb.Phi, pb.XL, pb.Y, pb.h, pb.sigma)
        B1, V1 = e.run_snps(pb.XR)
        with pytest.raises(FGLSError):
            e.set_problem(bad, pb.XL, pb.Y, pb.h, pb.sigma)
        e.set_problem(pb.Phi, pb.XL, pb.Y, pb.h, pb.sigma)
        B2, V2 = e.run_snps(pb.XR)
    assert np.array_equal(B1, B2) and np.array_equal(V1, V2)


@pytest.mark.parametrize("n", [200, 700])  # FP64 kernels, digits
@pytest.mark.parametrize("wXR", [1, 2])
def test_genotype_whose_square_overflows(n, wXR):
    """A value of 1e300 makes its SNP's quadratic term infinite and its own effect zero or
    NaN; the call is not refused, and the other SNPs are as without it."""
    from fgls_gb300 import Engine, datagen
    pb = datagen.make_problem(n, 256, 2, wXR=wXR, seed=n, hsig_uniform=True)
    X = pb.XR.copy()
    X[13, 7 * wXR] = 1e300
    with Engine(n, 3, wXR, 2, 256, variant="eigen") as e:
        e.set_problem(pb.Phi, pb.XL, pb.Y, pb.h, pb.sigma)
        B0, V0 = e.run_snps(pb.XR)
        B, V = e.run_snps(X)
    others = np.arange(256) != 7
    assert np.array_equal(B[:, others], B0[:, others]) and np.array_equal(V[:, others], V0[:, others])
    assert np.isfinite(B[:, 7, :3]).all()
