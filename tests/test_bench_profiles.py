"""The DRAM bytes per launch that bench.py takes from the committed ncu summaries."""
import os
import re

from conftest import ROOT


def test_bench_reads_summaries_whose_sum_is_their_own_counters():
    """Every summary bench.py names, at its default sizes (n = 10000, t = 100, 16384 SNPs;
    64 cohorts, 2048 SNPs), exists, and the line bench.py reads is the sum of the read and
    write counters that the file lists."""
    import bench
    names = re.findall(r'gemm_traffic\(f"([^"]+)"\)', open(os.path.join(ROOT, "bench.py")).read())
    assert len(names) == 2
    sizes = {"n": 10000, "t": 100, "xb": 16384, "C": 64}
    for name in names:
        at = dict(sizes, xb=2048) if "cohorts" in name else sizes
        name = re.sub(r"\{(\w+)\}", lambda m: str(at[m.group(1)]), name)
        text = open(os.path.join(ROOT, "profiles", name + ".txt")).read()
        both = sum(float(re.search(r"dram__bytes_%s\.sum\s+([\d.]+) GB" % k, text).group(1)) for k in ("read", "write"))
        assert abs(bench.gemm_traffic(name) - both * 1e9) < 0.02e9, name
