"""Bounded waits of the FP64 path's digit products (csrc/fgls_digit_gemm.cu): with a
limit of 1 ns the kernel gives up at its first wait that does not complete at once,
lets its copies and MMAs finish (those waits keep the 2 s limit), frees its TMEM and
returns; the call that launched it reports FGLSGPU_ETIMEOUT, and with the default
limit restored the same engine gives bit-identical results."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("variant,wXR", [("eigen", 1), ("eigen", 2), ("chol", 1)])
def test_expired_wait_in_a_block(variant, wXR):
    from fgls_gb300 import Engine, FGLSError, datagen
    from fgls_gb300.engine import ETIMEOUT
    pb = datagen.make_problem(1000, 400, 2, wXR=wXR, seed=5, hsig_uniform=True)  # two blocks, the second ragged
    with Engine(pb.n, pb.wXL, wXR, pb.t, 256, variant=variant) as e:
        e.set_problem(pb.Phi, pb.XL, pb.Y, pb.h, pb.sigma)
        e.select_trait(0)
        B1, V1 = e.run_snps(pb.XR)
        e.set_wait_limit(1)
        with pytest.raises(FGLSError) as ei:
            e.run_snps(pb.XR)
        assert ei.value.code == ETIMEOUT and "wait expired" in str(ei.value), ei.value
        e.set_wait_limit(0)
        B2, V2 = e.run_snps(pb.XR)
    assert np.array_equal(B1, B2) and np.array_equal(V1, V2)


def test_expired_wait_in_the_read_of_the_adjoint():
    """dY = Z V2 is launched by the read itself (n = 2000, t = 32: on digits)."""
    import torch
    from fgls_gb300 import Engine, FGLSError, datagen
    from fgls_gb300.engine import ETIMEOUT
    pb = datagen.make_problem(2000, 256, 32, seed=6, hsig_uniform=True)
    bbar = torch.from_numpy(np.random.default_rng(6).standard_normal((pb.t, pb.m, pb.p))).cuda()
    X = torch.from_numpy(np.ascontiguousarray(pb.XR.T)).cuda()
    torch.cuda.synchronize()
    with Engine(pb.n, pb.wXL, 1, pb.t, 256, variant="eigen") as e:
        e.set_problem(pb.Phi, pb.XL, pb.Y, pb.h, pb.sigma)
        e.adjoint_reset()
        e.adjoint_block_device(X.data_ptr(), pb.m, bbar.data_ptr(), bbar.stride(0))
        first = e.adjoint_read()
        e.set_wait_limit(1)
        with pytest.raises(FGLSError) as ei:
            e.adjoint_read()
        assert ei.value.code == ETIMEOUT, ei.value
        e.set_wait_limit(0)
        again = e.adjoint_read()
    for a, b in zip(first, again):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("call", ["set_hsigma", "set_precision"])
def test_expired_wait_in_the_split_operands(call):
    """U = Z [d y, d XL] (n = 1000, 160 columns: on digits) is the last product of
    the calls that build the split path's operands; with given slices no probe
    block follows it."""
    from fgls_gb300 import Engine, FGLSError, datagen
    from fgls_gb300.engine import ETIMEOUT
    pb = datagen.make_problem(1000, 200, 40, seed=7, hsig_uniform=True)
    first = "split" if call == "set_hsigma" else "fp64"
    with Engine(pb.n, 3, 1, pb.t, 256, variant="eigen", precision="split", slices=9) as e:
        e.set_problem(pb.Phi, pb.XL, pb.Y, pb.h, pb.sigma)
        B1, V1 = e.run_snps(pb.XR)
    with Engine(pb.n, 3, 1, pb.t, 256, variant="eigen", precision=first, slices=9) as e:
        def build():
            if call == "set_hsigma":
                e.set_hsigma(pb.h, pb.sigma)
            else:
                e.set_precision("split")
        e.set_problem(pb.Phi, pb.XL, pb.Y, pb.h, pb.sigma)
        e.set_wait_limit(1)
        with pytest.raises(FGLSError) as ei:
            build()
        assert ei.value.code == ETIMEOUT, ei.value
        e.set_wait_limit(0)
        if call == "set_hsigma":  # the problem's operands are gone, as after any failure of the call
            e.set_problem(pb.Phi, pb.XL, pb.Y, pb.h, pb.sigma)
        build()
        B2, V2 = e.run_snps(pb.XR)
    assert np.array_equal(B1, B2) and np.array_equal(V1, V2)


def test_expired_wait_in_an_eigendecomposition_that_fails():
    """A NaN in Phi makes the QL iteration fail as well: the expired wait is the
    error, and it is not left for the next call to report."""
    from fgls_gb300 import Engine, FGLSError, datagen
    from fgls_gb300.engine import ETIMEOUT
    pb = datagen.make_problem(1100, 64, 2, seed=8, hsig_uniform=True)
    bad = pb.Phi.copy()
    bad[5, 9] = bad[9, 5] = np.nan
    with Engine(pb.n, 3, 1, 2, 64, variant="eigen") as e:
        e.set_wait_limit(1)
        with pytest.raises(FGLSError) as ei:
            e.set_problem(bad, pb.XL, pb.Y, pb.h, pb.sigma)
        assert ei.value.code == ETIMEOUT, ei.value
        e.set_wait_limit(0)
        e.set_problem(pb.Phi, pb.XL, pb.Y, pb.h, pb.sigma)
        e.run_snps(pb.XR)


def test_expired_wait_in_the_inverse_when_the_block_digits_do_not_fit():
    """n = 762: of select_trait's products only those of L^-1 run on digits.  The digits
    of a block of 65536 SNPs (600 MB) do not fit, which must not lose their error."""
    import torch
    from fgls_gb300 import Engine, FGLSError, datagen
    from fgls_gb300.engine import ETIMEOUT
    pb = datagen.make_problem(762, 300, 1, seed=9, hsig_uniform=True)
    with Engine(pb.n, 3, 1, 1, 300, variant="chol") as e:
        e.set_problem(pb.Phi, pb.XL, pb.Y, pb.h, pb.sigma)
        e.select_trait(0)
        B1, V1 = e.run_snps(pb.XR)
    with Engine(pb.n, 3, 1, 1, 65536, variant="chol") as e:
        e.set_problem(pb.Phi, pb.XL, pb.Y, pb.h, pb.sigma)
        free, _ = torch.cuda.mem_get_info()
        fill = torch.empty(free - (320 << 20), dtype=torch.uint8, device="cuda")
        try:
            e.set_wait_limit(1)
            with pytest.raises(FGLSError) as ei:
                e.select_trait(0)
            assert ei.value.code == ETIMEOUT, ei.value
            e.set_wait_limit(0)
            e.select_trait(0)
            B2, V2 = e.run_snps(pb.XR)
        finally:
            del fill
            torch.cuda.empty_cache()
    # two FP64-accurate routes of the same problem, as in test_gpu_scratch_limits.py
    i = np.arange(pb.p)
    se = np.abs(V1[..., i, i])
    assert np.max(np.abs(B1 - B2) / (np.abs(B1) + se)) <= 1e-12
    assert np.max(np.abs(np.abs(V2[..., i, i]) - se) / se) <= 1e-12
