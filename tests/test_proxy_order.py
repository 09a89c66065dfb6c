"""The queue kernel of a ragged batch writes an array's rows twice in one launch: its column strips with
ordinary stores, its row blocks with bulk stores (the async proxy), from other CTAs.  The wait for the
strips orders the former among ordinary accesses only, so a proxy fence that covers global memory has to
stand between it and the bulk stores."""
import re
from pathlib import Path

CSRC = Path(__file__).resolve().parents[1] / "bridct_b200" / "csrc"


def test_row_blocks_of_the_queue_fence_the_proxies_after_their_wait():
    code = re.sub(r"//[^\n]*", "", (CSRC / "ragged.cuh").read_text())
    kernel = code[code.index("k_ragged(RaggedArgs a)"):]
    acquire = kernel.index("ld.acquire.gpu")
    barrier = kernel.index("__syncthreads()", acquire)
    rows = kernel.index("ragged_row_pass(", barrier)
    between = kernel[barrier:rows]
    assert re.search(r"fence\.proxy\.async(\.global)?;", between)
    # executed by every thread that issues a bulk store: not under a condition on the thread
    assert "threadIdx" not in between[:between.index("fence.proxy.async")]
