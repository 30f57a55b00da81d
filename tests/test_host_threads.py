"""Host threads of the network's graph join take no memory.

An exception that leaves a thread of a parallel region ends the process, where the
call should return an error. A failed allocation cannot be staged there, so this reads
the source.
"""
import re
from pathlib import Path

SOURCE = Path(__file__).resolve().parents[1] / "jump-cannon_b200" / "csrc" / "jc_mpnn.cu"


def _block(text, i):
    depth = 0
    for k in range(text.index("{", i), len(text)):
        depth += (text[k] == "{") - (text[k] == "}")
        if depth == 0:
            return text[i : k + 1]
    raise AssertionError("unbalanced")


def test_join_threads_take_no_memory():
    text = re.sub(r"//[^\n]*", "", SOURCE.read_text())
    join = _block(text, text.index("HostSet assemble("))
    loops = [_block(join, m.end()) for m in re.finditer(r"#pragma omp parallel for[^\n]*", join)]
    assert len(loops) == 2
    for loop in loops:
        assert not re.search(r"push_back|emplace|insert\(|resize\(|reserve\(|std::string|std::vector|\bnew\b|\bfail\(", loop)


def test_no_exception_leaves_the_no_allocation_pass():
    """Its launches throw on failure; any exception has to become a status."""
    text = re.sub(r"//[^\n]*", "", (SOURCE.parent / "jc_fa2.cu").read_text())
    entry = _block(text, text.index('extern "C" jc_status jc_fa2_bh_forces_noalloc('))
    assert "launch_chained(" in entry
    assert "catch (...)" in entry
