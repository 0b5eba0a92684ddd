"""Order of mbarrier set-up and waits in the stencil kernel, read from its
source: a lane that polls a barrier before it is initialised may read a box
that has not arrived.  That cannot be shown on a GPU (it depends on how the
compiler lets a warp reconverge), so the text is held to it."""
import os
import re

SRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "uq_b200", "csrc", "lbm_flux.cuh")


def _block(src, at):
    """src[at] is an opening brace: the index after the one that closes it."""
    depth = 0
    for k in range(at, len(src)):
        depth += (src[k] == "{") - (src[k] == "}")
        if depth == 0:
            return k + 1
    raise AssertionError("unbalanced braces")


def test_every_lane_is_ordered_after_its_warps_barrier_init():
    src = re.sub(r"//[^\n]*", "", open(SRC).read())
    kernel = src[src.index(" k_flux(KArgs<S> a)"):]
    kernel = kernel[:_block(kernel, kernel.index("{"))]
    inits = [m.start() for m in re.finditer(r"if \((?:lane|tid) == 0\) \{\s*(?:const int ix|for \(int b = 0)", kernel)]
    assert len(inits) == 2 and len(re.findall(r"\bmbar_init\(", kernel)) == 3
    # per warp: a warp barrier on every path, directly after the branch of lane 0
    after = kernel[_block(kernel, kernel.index("{", inits[0])):]
    assert after.lstrip().startswith("__syncwarp();"), after[:80]
    # one thread for the block (other tile shapes): the block barrier that those take
    barrier = re.search(r"if \(!TC \|\| [^\n]*\) __syncthreads\(\);", kernel)
    assert barrier and inits[1] < barrier.start() < kernel.index("sweep_tile<S>(")
    assert barrier.start() < kernel.index("mbar_wait_bounded(")
