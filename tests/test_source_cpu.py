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


def loads_from_tensor_memory():
    """(file, line number, array, the code after the load) of every tmem_ld call outside its definition."""
    for f in sorted(os.listdir(CSRC)):
        text = re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, f)).read())
        for m in re.finditer(r"(?<!void )\btmem_ld(?:4|16|32|32_if)\(", text):
            depth, end = 1, m.end()
            while depth:
                depth += {"(": 1, ")": -1}.get(text[end], 0)
                end += 1
            array = re.search(r"(\w+(?:\[\w+\])?)\)*$", text[m.end():end - 1].strip()).group(1)
            yield f, text.count("\n", 0, m.start()) + 1, array, text[end:]


def test_what_is_loaded_from_tensor_memory_is_waited_for_by_name():
    """tcgen05.ld is asynchronous: until the wait its registers hold nothing, and neither the order of statements nor a memory
    clobber keeps arithmetic on them behind it. Each array goes through the wait that covers it before anything else names it, on
    a straight way: no branch, loop or end of a block in between."""
    loads = list(loads_from_tensor_memory())
    assert len(loads) >= 10, loads
    for f, line, array, after in loads:
        name = re.escape(array.split("[")[0])
        wait = re.search(r"\btmem_ld_wait\(([^()]*)\);", after)
        assert wait and array in [a.strip() for a in wait.group(1).split(",")], f"{f}:{line}: {array} is not what the next wait names"
        between = [s for s in after[:wait.start()].split(";") if "tmem_ld" not in s]
        assert not any(re.search(rf"\b{name}\b|\b(if|for|while|break|continue|return)\b|[{{}}]", s) for s in between), f"{f}:{line}: {between}"
