"""Kernels launched as programmatic dependents read the chain's data by ordinary loads.

A dependent is resident while the kernels before it still store, so what they
write is not read-only for its lifetime: neither __ldg nor ld.global.nc may read
it, nor a __restrict__ pointer, which lets the compiler use them and move a load
above the wait. The fault cannot be made to show on a GPU at will, so this reads
the sources: each chained kernel may hold __restrict__ pointers (and __ldg
operands) only for data that no kernel of its chain writes before it.
"""
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "jump-cannon_b200" / "csrc"
TEXT = {p.name: re.sub(r"//[^\n]*", "", p.read_text()) for p in sorted(CSRC.iterdir()) if p.suffix in (".cu", ".cuh")}

# kernel -> parameters no earlier kernel of its chain writes: graphs, degrees,
# items, the per-pair engine's drawn samples and its schedule, and the positions
# (moved by the last kernel of a step, after which the next chain begins anew).
READ_ONLY = {
    "k_keys": {"pos"},
    "os_pass": set(),
    "k_seg_fix": set(),
    "k_count": set(),
    "k_offsets": set(),
    "k_fill": {"pos", "degf"},
    "k_com_kids": set(),
    "k_walk_ahead": {"pos", "degf"},
    "k_walk_warp": {"pos", "degf"},
    "k_att": {"order", "off", "nbr", "pos", "old_force", "degf"},
    "k_apply": {"degf"},
    "k_smooth": set(),
    "k_smooth_hub": {"hubs"},
    "k_proj_center_sums": {"deg", "items"},
    "k_center_coef": {"item_off", "go"},
    "k_proj_center": set(),
    "k_pairs": {"samples", "eta_table", "sweep_ctr"},
    "k_pairs_apply": {"samples"},
}
# operands of __ldg in device functions of those kernels: the CSR, and the
# positions of the attraction pass
LDG = {"row", "nbr", "pos"}


def _balanced(s, i, pair):
    depth = 0
    for k in range(i, len(s)):
        depth += (s[k] == pair[0]) - (s[k] == pair[1])
        if depth == 0:
            return k
    raise AssertionError("unbalanced")


def _functions():
    """name -> [(parameters, body)] of every __global__ / __device__ function."""
    out = {}
    for text in TEXT.values():
        text = re.sub(r"__launch_bounds__\((?:[^()]|\([^()]*\))*\)", "", text)
        for m in re.finditer(r"__(?:global|device)__\s+(?:[\w:<>*&]+\s+)+?(\w+)\s*\(", text):
            i = m.end() - 1
            j = _balanced(text, i, "()")
            k = j + 1
            while k < len(text) and text[k].isspace():
                k += 1
            if k < len(text) and text[k] == "{":
                out.setdefault(m.group(1), []).append((text[i + 1 : j], text[k : _balanced(text, k, "{}") + 1]))
    return out


FUNCTIONS = _functions()


def _chained():
    names = set()
    for text in TEXT.values():
        for m in re.finditer(r"\blaunch_chained\s*\(", text):
            i = m.end() - 1
            call = text[i : _balanced(text, i, "()")]
            names |= set(re.findall(r"\b(k_\w+)\b", call))
            if re.search(r"\bpass\b", call):  # radix_passes picks os_pass by size
                names.add("os_pass")
    return names


def test_every_chained_kernel_is_listed():
    assert _chained() == set(READ_ONLY)


@pytest.mark.parametrize("kernel", sorted(READ_ONLY))
def test_chained_kernel_reads(kernel):
    assert kernel in FUNCTIONS, "kernel not found in the sources"
    seen, todo = set(), [kernel]
    while todo:  # the kernel and every device function it reaches
        f = todo.pop()
        if f in seen:
            continue
        seen.add(f)
        for params, body in FUNCTIONS[f]:
            if f == kernel:
                got = set(re.findall(r"__restrict__\s+(\w+)", params))
                assert got <= READ_ONLY[kernel], f"{kernel}: __restrict__ on {sorted(got - READ_ONLY[kernel])}"
                assert "dependent_launch_wait" in body
            assert "global.nc" not in body, f"{kernel} -> {f}: read-only load"
            for arg in re.findall(r"__ldg\(\s*(?:reinterpret_cast<[^>]*>\(\s*)?(\w+)", body):
                assert arg in LDG, f"{kernel} -> {f}: __ldg({arg} ...)"
            calls = set(re.findall(r"\b(\w+)\s*(?:<[^<>;(){}]*>)?\s*\(", body)) & set(FUNCTIONS)
            # the read-only walk of the unchained launches shares walk_one
            if f == "walk_one" and re.search(r"if \(CHAINED\) load_node_c\(.*?;\s*else load_node\(", body):
                calls.discard("load_node")
            todo += calls


# A sort that gave up waiting leaves a permutation (and a batch's sorted keys) that may
# hold anything: the kernels behind it read neither once the error word is set.
@pytest.mark.parametrize("kernel,reads", [("k_walk", "order["), ("k_walk_ahead", "order["), ("k_walk_rope", "order["),
                                          ("k_walk_top", "order["), ("k_walk_warp", "order["), ("k_fill", "val["),
                                          ("k_graph_trees", "hi[a]")])
def test_no_permutation_is_followed_after_an_error(kernel, reads):
    (_, body), = FUNCTIONS[kernel]
    checked, previous = False, ""
    for line in body[: body.rindex(reads) + len(reads)].splitlines():
        checked |= bool(re.search(r"if \(.*st->error.*\) return;", line))
        if reads in line:
            assert checked or "!failed" in line or "!failed" in previous, line
        previous = line or previous
