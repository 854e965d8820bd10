"""Device memory that the digits of the FP64 products take: only where a call uses
them, and not from calls that fit without."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

MB = 1 << 20


def free_bytes():
    import torch
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    return torch.cuda.mem_get_info()[0]


class Fill:
    """Takes the device's memory but `left` bytes."""

    def __init__(self, left):
        import torch
        free = free_bytes()
        assert free > left
        self.t = torch.empty(free - left, dtype=torch.uint8, device="cuda")

    def __enter__(self):
        return self

    def __exit__(self, *exc):
        import torch
        del self.t
        torch.cuda.empty_cache()


def same(B, V, B0, V0):
    """Two FP64-accurate routes of one problem: 1e-12 on the standard errors' scale, as for parity."""
    i = np.arange(B.shape[-1])
    se = np.abs(V0[..., i, i])
    assert np.max(np.abs(B - B0) / (np.abs(B0) + se)) <= 1e-12
    assert np.max(np.abs(np.abs(V[..., i, i]) - se) / se) <= 1e-12


def test_split_chol_takes_no_digits_of_a_whole_block():
    """The split path's blocks have operands of their own; its FP64 probe block takes the
    digits of 256 SNPs.  Those of a whole block (16384 SNPs: 590 MB) do not fit here, and
    the next trait's set-up must not notice."""
    from fgls_gb300 import Engine, datagen
    from fgls_gb300.engine import launch_count
    n = 3000
    pb = datagen.make_problem(n, 64, 2, seed=10)
    pb.Y[:, 1] = pb.Y[:, 0]  # the same trait twice: the same launches
    with Engine(n, 3, 1, 2, 16384, variant="chol", precision="split") as e:
        def launches(j):
            a = launch_count()
            e.select_trait(j)
            return launch_count() - a
        e.set_problem(pb.Phi, pb.XL, pb.Y, pb.h, pb.sigma)
        e.select_trait(0)  # the plan
        usual = launches(1)
        with Fill(500 * MB):
            launches(0)
            assert launches(1) == usual


def test_chol_traits_after_the_digits_were_given_back():
    """The widened genotypes (524 MB) take the digits' place; the next select_trait must
    not take L^-1 (128 MB) and the digits (980 MB) again, which its blocks will not use."""
    from fgls_gb300 import Engine, datagen
    n = 4000
    pb = datagen.make_problem(n, 64, 2, seed=11, hsig_uniform=True)
    G = np.ascontiguousarray(np.tile(pb.XR.astype(np.uint8), (1, 4)).T)
    with Engine(n, 3, 1, 2, 16384, variant="chol") as e:
        e.set_problem(pb.Phi, pb.XL, pb.Y, pb.h, pb.sigma)
        ref = []
        for j in range(2):
            e.select_trait(j)
            ref.append(e.run_block(pb.XR))
        with Fill(384 * MB):
            e.run_snps_genotypes(G)
        before = free_bytes()
        for j in range(2):
            e.select_trait(j)
            same(*e.run_block(pb.XR), *ref[j])
        assert before - free_bytes() < 64 * MB  # the factorization's own panels


@pytest.mark.parametrize("variant", ["eigen", "chol"])
def test_split_set_up_gives_its_operands_back(variant):
    """A split engine of 9 given slices holds no more than one that chose its 9 by the
    probe: the digits of the set-up's FP64 products (two operands of 108 MB) go."""
    from fgls_gb300 import Engine, datagen
    pb = datagen.make_problem(3000, 64, 40, seed=12, hsig_uniform=True)
    held = {}
    for slices in (9, 0):
        before = free_bytes()
        with Engine(pb.n, 3, 1, 40, 256, variant=variant, precision="split", slices=slices) as e:
            e.set_problem(pb.Phi, pb.XL, pb.Y, pb.h, pb.sigma)
            e.select_trait(0)
            held[slices] = before - free_bytes()
    assert held[9] <= held[0] + 16 * MB, held


@pytest.mark.parametrize("variant", ["eigen", "chol"])
def test_no_workspace_in_small_engines(variant):
    """The digit products' workspace (120 MB) is taken by the first product on digits."""
    from fgls_gb300 import Engine, datagen
    n = 150
    pb = datagen.make_problem(n, 64, 2, seed=13, hsig_uniform=True)
    for _ in range(2):  # the first time the device also loads the kernels
        before = free_bytes()
        with Engine(n, 3, 1, 2, 64, variant=variant) as e:
            e.set_problem(pb.Phi, pb.XL, pb.Y, pb.h, pb.sigma)
            e.select_trait(0)
            e.run_block(pb.XR)
            held = before - free_bytes()
    assert held < 48 * MB


def test_split_engine_gives_its_workspace_back():
    """A split engine's blocks use no digits; the workspace of its set-up goes to the FP64
    path's buffers (two of 49 MB) where the device has no other room."""
    from fgls_gb300 import Engine, datagen
    pb = datagen.make_problem(3000, 64, 2, seed=13, hsig_uniform=True)
    with Engine(pb.n, 3, 1, 2, 2048, variant="eigen", precision="split") as e:
        e.set_problem(pb.Phi, pb.XL, pb.Y, pb.h, pb.sigma)
        with Fill(64 * MB):
            e.set_precision("fp64")
            B, V = e.run_block(pb.XR)
    with Engine(pb.n, 3, 1, 2, 64, variant="eigen") as e:
        e.set_problem(pb.Phi, pb.XL, pb.Y, pb.h, pb.sigma)
        same(B, V, *e.run_block(pb.XR))



def test_split_plan_holds_the_pass_sums_of_its_own_tiles():
    """512 KB a CTA that the block launches (n = 300, 64 SNPs: two pairs), not one per SM."""
    from fgls_gb300 import Batch, Engine, datagen
    from test_gpu_batch import run_batch
    pb = datagen.make_problem(300, 64, 2, seed=14, hsig_uniform=True)
    desc = [{"Phi": pb.Phi, "XL": pb.XL, "Y": pb.Y, "h": pb.h, "sigma": pb.sigma}]
    for _ in range(2):  # the first time the device also loads the kernels
        held = []
        for variant in ("eigen", "chol"):
            before = free_bytes()
            with Engine(pb.n, 3, 1, 2, 64, variant=variant, precision="split", slices=9) as e:
                e.set_problem(pb.Phi, pb.XL, pb.Y, pb.h, pb.sigma)
                e.select_trait(0)
                e.run_block(pb.XR)
                held.append(before - free_bytes())
        before = free_bytes()
        with Batch(desc, x_b=64, slices=9) as b:
            held.append(before - free_bytes())
            run_batch(b, [pb], 64)
    assert max(held) < 48 * MB, held


@pytest.mark.parametrize("second", ["eigen", "chol", "batch"])
def test_another_engine_fits_in_the_digits_place(second):
    """The digits of one engine's blocks (590 MB and 108 MB of Z) give way to a second
    engine or batch on the device that fits without them."""
    from fgls_gb300 import Batch, Engine, datagen
    from test_gpu_batch import run_batch
    n, x_b = 3000, 16384
    pb = datagen.make_problem(n, 64, 1, seed=15, hsig_uniform=True)
    desc = [{"Phi": pb.Phi, "XL": pb.XL, "Y": pb.Y, "h": pb.h, "sigma": pb.sigma}]

    class Second:
        def __enter__(self):
            if second == "batch":
                self.b = Batch(desc, x_b=8192, slices=9)
            else:
                self.b = Engine(n, 3, 1, 1, 8192, variant=second)
                self.b.set_problem(pb.Phi, pb.XL, pb.Y, pb.h, pb.sigma)
                self.b.select_trait(0)
            return self

        def run(self):
            return run_batch(self.b, [pb], 64)[0] if second == "batch" else self.b.run_block(pb.XR)

        def __exit__(self, *exc):
            self.b.close()

    # what the second holds or needs while it is set up, no more: its own digits left out
    # (megabytes of matrices, blocks, divide and conquer; of operands, output and scratch)
    need = {"eigen": 3 * 72 + 4 * 197 + 288 + 5, "chol": 2 * 72 + 3 * 197,
            "batch": 25 + 85 + 207 + 4 * 72 + 12}[second] * MB
    with Second() as s:
        ref2 = s.run()
    with Engine(n, 3, 1, 1, x_b, variant="eigen") as e:
        e.set_problem(pb.Phi, pb.XL, pb.Y, pb.h, pb.sigma)
        ref = e.run_block(pb.XR)
        with Fill(need - 300 * MB):
            with Second() as s:
                same(*e.run_block(pb.XR), *ref)
                tol = 1e-10 if second == "batch" else 1e-12
                out = s.run()
        i = np.arange(pb.p)
        se = np.abs(ref2[1][..., i, i])
        assert np.max(np.abs(out[0] - ref2[0]) / (np.abs(ref2[0]) + se)) <= tol


def test_engines_on_two_threads_while_memory_is_short():
    """One thread runs blocks while another creates and sets up engines that need the
    first one's digits: every block is right, whatever the timing."""
    import threading
    from fgls_gb300 import Engine, FGLSError, datagen
    n, x_b = 3000, 16384
    pb = datagen.make_problem(n, 64, 1, seed=16, hsig_uniform=True)
    with Engine(n, 3, 1, 1, x_b, variant="eigen") as e:
        e.set_problem(pb.Phi, pb.XL, pb.Y, pb.h, pb.sigma)
        ref = e.run_block(pb.XR)
        stop, bad = threading.Event(), []

        def blocks():
            try:
                while not stop.is_set():
                    same(*e.run_block(pb.XR), *ref)
            except BaseException as x:  # noqa: BLE001
                bad.append(x)
        t = threading.Thread(target=blocks)
        with Fill(1200 * MB):
            t.start()
            made = 0
            try:
                for _ in range(200):
                    if made == 5:
                        break
                    try:
                        with Engine(n, 3, 1, 1, 8192, variant="eigen") as o:
                            o.set_problem(pb.Phi, pb.XL, pb.Y, pb.h, pb.sigma)
                            same(*o.run_block(pb.XR), *ref)
                            made += 1
                    except FGLSError as x:  # refused while the other engine is in a call
                        assert "memory" in str(x), x
            finally:
                stop.set()
                t.join()
    assert not bad, bad
    assert made > 0
