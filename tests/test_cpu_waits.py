"""Every wait of a kernel is bounded: what the sources may and may not use to wait.

A wait that has run out lets its warp leave the loop on its own, so nothing that waits without a limit may stand where such a
warp is missed.  A kernel that hangs cannot be made to fail on purpose on a GPU, so this reads the sources."""
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "zenith_b200" / "csrc"
SOURCES = {p.name: re.sub(r"//[^\n]*", "", p.read_text()) for p in sorted([*CSRC.glob("*.cu"), *CSRC.glob("*.cuh")])}


@pytest.mark.parametrize("name", SOURCES)
def test_no_named_barriers(name):
    """Warps of a group meet at an mbarrier (``mbar_wait`` has a limit), never at ``bar.sync`` / ``barrier.sync``."""
    assert not re.search(r"\bbar(rier)?\.(cta\.)?(sync|arrive|red)\b", SOURCES[name])


@pytest.mark.parametrize("name", [n for n in SOURCES if n != "zen_common.cuh"])
def test_mbarriers_are_polled_with_a_limit(name):
    """``mbarrier.try_wait`` / ``test_wait`` stand only in the helpers that ``mbar_wait`` and ``mbar_wait_cluster`` bound."""
    assert not re.search(r"mbarrier\.(try|test)_wait|mbar_try_wait", SOURCES[name])


@pytest.mark.parametrize("name", ["gemm_small.cuh", "gemm_ln.cu", "gemm_pair.cuh"])
def test_a_cta_leaves_its_shared_memory_after_its_peers_are_through_with_it(name):
    """A CTA whose waits have run out has not seen all that its peers write to it: the tear-down of a kernel with such writes
    (behind its last ``__syncthreads``) holds a wait for every CTA of the cluster."""
    text = SOURCES[name]
    writes = [m.end() for m in re.finditer(r"map_to_cta\(", text)]
    body = text[writes[-1]:]
    tear_down = body[body.index("__syncthreads();"):]
    assert re.search(r"cluster_(leave|sync_all)\(", tear_down[:tear_down.index("\n}\n")])


@pytest.mark.parametrize("name", [n for n in SOURCES if n not in ("zen_common.cuh", "selftest.cu")])
def test_the_lanes_of_a_warp_give_up_together(name):
    """``mbar_wait`` is for single threads (inside ``if (.. elect_one()) {``); warps wait with the ``_warp`` forms, whose lanes all
    get the same answer, as instructions of the whole warp follow."""
    text = SOURCES[name]
    elected = []
    for m in re.finditer(r"elect_one\(\)\) \{", text):
        depth, i = 1, m.end()
        while depth:
            depth += {"{": 1, "}": -1}.get(text[i], 0)
            i += 1
        elected.append((m.end(), i))
    for m in re.finditer(r"\bmbar_wait(_cluster)?\(", text):
        assert any(lo <= m.start() < hi for lo, hi in elected), text[m.start():m.start() + 80]
