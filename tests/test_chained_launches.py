"""Kernels launched before the one ahead of them ends (programmatic dependent launch)
read what that one is still writing: their pointers are not declared constant or
unaliased, which would let the compiler load through them ahead of the wait."""
import glob
import os
import re

from conftest import ROOT

CSRC = os.path.join(ROOT, "cugwas-proto_gb300", "csrc")


def test_no_constant_or_unaliased_pointers_in_chained_kernels():
    seen = 0
    for path in glob.glob(os.path.join(CSRC, "*.cu")):
        src = re.sub(r"//[^\n]*", "", open(path).read())
        for name in set(re.findall(r"launch_chained\((\w+_kernel)", src)):
            args = re.search(r"__global__[^;{]*?\b" + name + r"\(([^)]*)\)\s*\{", src).group(1)
            pointers = [a for a in args.split(",") if "*" in a]
            assert pointers
            for a in pointers:
                assert "__restrict__" not in a and "const" not in a, (name, a.strip())
            seen += 1
    assert seen >= 2
