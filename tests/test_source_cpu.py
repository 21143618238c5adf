"""What the kernels' sources must keep to, where no run could show it."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "et_b200", "csrc")


def test_a_warp_branches_on_a_barrier_only_by_a_bounded_wait_or_a_vote():
    """mbarrier.try_wait answers each lane for itself. A warp whose lanes branched on different answers would meet in different
    warp-wide operations, which no bounded wait ends: only mbar_wait and mbar_poll_warp may ask."""
    asks = [(f, line.strip()) for f in sorted(os.listdir(CSRC)) for line in open(os.path.join(CSRC, f)) if re.search(r"\bmbar_try_wait\(", line)]
    assert [f for f, _ in asks] == ["ptx.cuh"] * 3, asks
    assert sum("__all_sync" in line for _, line in asks) == 1, asks
