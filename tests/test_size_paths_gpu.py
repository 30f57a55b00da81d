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


# pivot counts around the groups of eight; both block shapes (up to 75,776
# nodes and above); distances beyond the (mu, d) table (a 5,000-node path); an
# eta below the in-range bound; nodes on top of a pivot and far from all
@pytest.mark.parametrize("case", ["k1", "k7", "k8", "k9", "n75776", "n75777", "path5000", "eta-tiny", "clamped-far"])
def test_jacobi_forms_bit_exact(jc, orc, case):
    s = {"n_pivots": 9, "eta_max": 2.0}
    steps = 3
    if case[0] == "k":
        g, s["n_pivots"] = jc.gen_scale_free(1500, 2, 5), int(case[1:])
    elif case[0] == "n":
        g, s["n_pivots"], steps = jc.gen_watts_strogatz(int(case[1:]), 4, 0.2, 3), 3, 2
    elif case == "path5000":
        g, s["eta_max"] = jc.gen_path(5000), 1.0e7
    else:
        g = jc.gen_grid(30)
        if case == "eta-tiny":
            s.update(eta_max=1.0e-7, eta_min=1.0e-8)
    pos = jc.seed_uniform(g.n_nodes, 3, 11) * np.float32(20.0)
    if case == "clamped-far":
        pos[:] = np.tile(pos[:3], g.n_nodes)     # all on one point: every magnitude clamped
        pos[3 * 50:3 * 60] += np.float32(1e-7)   # closer than the clamp
        pos[3 * 100:3 * 110] *= np.float32(1e12)  # squared distances past 2^60
    e = jc.LayoutEngine("sgd-stress-gpu")
    e.set_params(s)
    e.init(g, pos)
    o = orc.Sgd(g, pos, mode=1, **s)
    for _ in range(steps):
        assert np.array_equal(bits(e.step()), bits(o.step()))
    assert np.array_equal(bits(e.positions()), bits(o.positions()))
