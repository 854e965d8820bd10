"""The split GEMM's pass sums in either form (planes, int64 sums), at the lines of the
rule, with ragged rows, columns and blocks and odd and even slice counts, against the
FP64 path.  Each slice less multiplies the split path's 1e-10 by its base, 32."""
import numpy as np
import pytest

from conftest import report
from oracle import fgls_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [3968, 3969, 4097])  # padded K of 3968, 4096 and 4224
@pytest.mark.parametrize("t", [1, 40])
def test_split_against_fp64_around_the_line(n, t):
    from fgls_gb300 import Engine, datagen
    pb = datagen.make_problem(n, 301, t, seed=n, hsig_uniform=True, markers=3000)
    with Engine(n, 3, 1, t, 256, variant="eigen") as e:
        e.set_problem(pb.Phi, pb.XL, pb.Y, pb.h, pb.sigma)
        Br, Vr = e.run_snps(pb.XR)
    for S in (9, 8, 7):
        with Engine(n, 3, 1, t, 256, variant="eigen", precision="split", slices=S) as e:
            e.set_problem(pb.Phi, pb.XL, pb.Y, pb.h, pb.sigma)
            d = O.compare(*e.run_snps(pb.XR), Br, Vr)
        report(f"split_sums_n{n}_t{t}_s{S}", **d)
        tol = 1e-10 * 32.0 ** (9 - S)
        assert d["finite"] and d["beta_normwise"] <= tol and d["se_rel"] <= tol, (S, d)


@pytest.mark.parametrize("n", [1920, 1921])  # padded K of 1920 and 2048
def test_triangular_operand_of_one_wave(n):
    from fgls_gb300 import Engine, datagen
    pb = datagen.make_problem(n, 301, 1, seed=n, hsig_uniform=True)
    with Engine(n, 3, 1, 1, 256, variant="chol") as e:
        e.set_problem(pb.Phi, pb.XL, pb.Y, pb.h, pb.sigma)
        e.select_trait(0)
        Br, Vr = e.run_snps(pb.XR)
    for S in (9, 8, 7):
        with Engine(n, 3, 1, 1, 256, variant="chol", precision="split", slices=S) as e:
            e.set_problem(pb.Phi, pb.XL, pb.Y, pb.h, pb.sigma)
            e.select_trait(0)
            d = O.compare(*e.run_snps(pb.XR), Br, Vr)
        tol = 1e-10 * 32.0 ** (9 - S)
        assert d["finite"] and d["beta_normwise"] <= tol and d["se_rel"] <= tol, (S, d)
