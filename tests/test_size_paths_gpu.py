"""Kernel variants chosen by size, at the edges of the rules that choose them,
against the CPU oracle (bit for bit: every variant keeps the oracle's order of
roundings)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def bits(a):
    return np.ascontiguousarray(a, np.float32).view(np.uint32)


# one body; remainders of the 256-body chunks and of the 4, 8 and 16 bodies a
# block; both sides of the rules (592, 1,184)
@pytest.mark.parametrize("n", [1, 2, 5, 255, 256, 257, 592, 593, 1184, 1185, 2051])
def test_brute_sizes_bit_exact(jc, orc, n):
    g = jc.gen_scale_free(n, 3, n) if n > 4 else jc.gen_path(n)
    pos = jc.seed_uniform(n, 3, n + 1)
    if n > 300:  # a coincident pair (distance clamp, zero terms) and a far body
        pos[3 * 7:3 * 7 + 3] = pos[3 * 290:3 * 290 + 3]
        pos[:3] = [3.0e4, -2.0e4, 1.0e4]
    e = jc.LayoutEngine("fa2-brute")
    e.init(g, pos)
    o = orc.Fa2(g, pos, bh=False)
    for _ in range(2):
        e.step()
        o.step()
        f, st = e.forces()
        r = o.get()
        assert np.array_equal(bits(f), bits(r["force"]))
        assert np.array_equal(bits(st), bits(r["stats"]))
        assert np.array_equal(bits(e.positions()), bits(r["pos"]))
