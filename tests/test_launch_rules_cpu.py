"""Kernels that are launched before their predecessor has ended read what it writes: nothing in their source may tell the compiler that this
memory does not change while they run (const __restrict__ parameters, __ldg of anything but the planes that a table row points to)."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "nestquant_b200", "csrc")


def _strip(s):
    return re.sub(r"//[^\n]*", "", s)


def test_kernels_launched_early_have_no_read_only_promises():
    src = {os.path.basename(f): _strip(open(f).read()) for f in glob.glob(os.path.join(CSRC, "*.cu*"))}
    early = {}
    for f, s in src.items():
        for call in re.finditer(r"launch_dependent\(([^;]*);", s):
            for k in re.findall(r"\b\w+_kernel\b", call.group(1)):
                early.setdefault(f, set()).add(k)
    assert sum(len(k) for k in early.values()) >= 11, early
    for f, kernels in early.items():
        for k in kernels:
            heads = re.findall(r"__global__[^;{]*?\b" + k + r"\(([^{]*)\)\s*\{", src[f])
            assert len(heads) == 1, (f, k)
            assert "__restrict__" not in heads[0], (f, k)
            assert "grid_dependency_wait();" in src[f].split(k + "(", 1)[1], (f, k)
        planes = [a for a in re.findall(r"__ldg\(([^;]*)", src[f]) if not re.search(r"\b[JI]\.P\.\w+", a)]
        assert not planes, (f, planes)
    assert "__restrict__" not in src["nq_plan.cuh"]
