"""Warp-wide TMEM instructions (`tcgen05 ... .sync.aligned`) need a converged warp:
their wrappers in csrc/tc_tile.cuh start with a __syncwarp, whatever branch or
per-thread wait came before the call, and nothing issues them outside a wrapper."""
import os
import re

from conftest import ROOT

CSRC = os.path.join(ROOT, "pybrown_b200", "csrc")
ALIGNED = re.compile(r"tcgen05\.(alloc|dealloc|ld)\.\S*sync\.aligned")


def _functions(src):
    """(name, body) of every function defined at the left margin."""
    for m in re.finditer(r"^__device__ [^;{]*?(\w+)\([^;{]*\) \{\n(.*?)^\}", src, re.M | re.S):
        yield m[1], m[2]


def test_tmem_wrappers_converge_the_warp():
    with open(os.path.join(CSRC, "tc_tile.cuh")) as f:
        src = f.read()
    found = {}
    for name, body in _functions(src):
        m = ALIGNED.search(body)
        if m:
            found[name] = "__syncwarp();" in body[:m.start()]
    assert found == {"tmem_alloc": True, "tmem_dealloc": True, "tmem_ld32": True}
    assert len(ALIGNED.findall(src)) == 3


def test_no_other_source_issues_them():
    for f in sorted(os.listdir(CSRC)):
        if f != "tc_tile.cuh":
            with open(os.path.join(CSRC, f)) as h:
                assert not ALIGNED.search(h.read()), f
