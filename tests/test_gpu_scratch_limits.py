"""Calls that allocate after the digits of the FP64 products are laid out: with the
device nearly full the engine gives the digits back instead of refusing the call."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LEFT = 384 << 20  # bytes left free, less than each call below allocates


@pytest.mark.parametrize("variant,t", [("eigen", 2), ("chol", 1)])
def test_widened_genotypes_fit_in_the_digits_place(variant, t):
    import torch
    from fgls_gb300 import Engine, datagen
    x_b = 16384  # 16384 SNPs of 4000 values: 524 MB widened, 200 to 1000 MB of digits
    pb = datagen.make_problem(4000, 64, t, wXL=3, seed=8, hsig_uniform=True)
    X = np.tile(pb.XR.astype(np.uint8), (1, x_b // 64))
    with Engine(pb.n, 3, 1, t, x_b, variant=variant) as e:
        e.set_problem(pb.Phi, pb.XL, pb.Y, pb.h, pb.sigma)
        e.select_trait(0)
        B0, V0 = e.run_snps(np.asfortranarray(X.astype(np.float64)))
        torch.cuda.synchronize()
        free, _ = torch.cuda.mem_get_info()
        assert free > LEFT
        fill = torch.empty(free - LEFT, dtype=torch.uint8, device="cuda")
        try:
            B, V = e.run_snps_genotypes(np.ascontiguousarray(X.T))
        finally:
            del fill
            torch.cuda.empty_cache()
    # two FP64-accurate routes of the same problem: 1e-12 on the standard errors' scale, as for parity
    p = B0.shape[-1]
    i = np.arange(p)
    se = np.abs(V0[..., i, i])
    assert np.max(np.abs(B - B0) / (np.abs(B0) + se)) <= 1e-12
    assert np.max(np.abs(np.abs(V[..., i, i]) - se) / se) <= 1e-12


def test_batch_setup_fits_without_its_digits():
    """One cohort of 3000 with four traits on four streams: 0.34 GB of operands and 0.94 GB
    of FP64 scratch are needed; the digits' 0.86 GB on top are not."""
    import torch
    from fgls_gb300 import Batch, datagen
    from test_gpu_batch import run_batch
    pb = datagen.make_problem(3000, 64, 4, wXL=3, seed=9, hsig_uniform=True)
    desc = [{"Phi": pb.Phi, "XL": pb.XL, "Y": pb.Y, "h": pb.h, "sigma": pb.sigma}]
    with Batch(desc, x_b=256, slices=9) as b:
        (B0, V0), = run_batch(b, [pb], 64)
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    left = 1750 << 20
    free, _ = torch.cuda.mem_get_info()
    assert free > left
    fill = torch.empty(free - left, dtype=torch.uint8, device="cuda")
    try:
        b = Batch(desc, x_b=256, slices=9)
    finally:
        del fill
        torch.cuda.empty_cache()
    with b:
        (B, V), = run_batch(b, [pb], 64)
    # the split path's bound, as against the oracle
    i = np.arange(pb.p)
    se = np.abs(V0[..., i, i])
    assert np.max(np.abs(B - B0) / (np.abs(B0) + se)) <= 1e-10
    assert np.max(np.abs(np.abs(V[..., i, i]) - se) / se) <= 1e-10
