"""Hand-overs of tensor memory in the dense maps, read off the source: no run shows a fence that is missing."""
import os
import re

from cbm4gnn_b200 import _lib

CSRC = os.path.join(os.path.dirname(_lib.__file__), "csrc")


def _source(name):
    return re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, name)).read())


def test_every_wait_is_followed_by_the_fence():
    """What a warp does in tensor memory behind an mbarrier (the store into a slot that MMAs have read, too) is
    ordered by ``tcgen05.fence::after_thread_sync``: the wait itself issues it, and there is no other wait."""
    wait = re.search(r"bool warp_wait\(.*?\n}\n", _source("cbm_map.cuh"), re.S).group(0)
    assert wait.index("bar_poll(") < wait.index("fence_after();")
    for name in ("cbm_map.cu", "cbm_map_grad.cu"):
        kernels = _source(name)
        polls = re.findall(r"bar_poll\((\w+)", kernels)
        assert polls == ["drained"]  # before the memory is freed: nothing is accessed behind it
        assert len(re.findall(r"warp_wait\(", kernels)) >= 4
