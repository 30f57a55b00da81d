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


def star(jc, leaves, extra):
    """A star with a path through its first `extra` leaves."""
    pairs = [(0, k) for k in range(1, leaves + 1)] + [(k, k + 1) for k in range(1, extra)]
    return jc.csr_from_pairs(leaves + 1, np.array(pairs, np.uint32))


# rows around the 32-entry rule of the long-row warps, their 16- and 32-entry
# chunks and the 1,024-entry hub rule; the oracle sums every row in the device's
# order and rounds to bf16 where the device stores bf16, so features may differ
# by a bf16 step of a flipped rounding and the rest by the bars of a bf16 network
@pytest.mark.parametrize("leaves", [31, 32, 33, 48, 63, 64, 65, 257, 1023, 1024, 1025])
def test_mpnn_row_lengths(jc, orc, leaves):
    graphs = [jc.gen_watts_strogatz(70, 6, 0.1, 3), star(jc, leaves, 20), jc.gen_scale_free(300, 3, 5)]
    rng = np.random.default_rng(7)
    targets = [rng.standard_normal(3 * g.n_nodes).astype(np.float32) for g in graphs]
    for t in targets:
        t[2::3] = 0.0
    net = jc.Mpnn(2, 99)
    net.set_params({"smooth_steps": 9, "cheb_steps": 17})
    net.bind(graphs, targets)
    gs = orc.GraphSet(graphs)
    X, xo = net.features(), orc.mpnn_features(gs, 99, smooth_steps=9, cheb_steps=17)
    assert np.array_equal(X[:, 1:17], xo[:, 1:17])
    assert np.all(np.abs(X[:, 17:25] - xo[:, 17:25]) <= 2.0 ** -6 * np.abs(xo[:, 17:25]) + 1e-5)
    loss, y, grad = net.grad(0, 3, pair_step=1)
    t4 = np.concatenate([np.concatenate([t.reshape(-1, 3), np.zeros((len(t) // 3, 1), np.float32)], 1) for t in targets])
    loss_o, y_o, grad_o = orc.mpnn_grad(gs, X, t4, 2, net.weights(), 8, 99, 1, 0, 3, emulate=True)
    assert loss == pytest.approx(loss_o, rel=1e-3)
    assert np.linalg.norm(y[:, :2] - y_o[:, :2]) <= 1e-2 * np.linalg.norm(y_o[:, :2])
    assert np.linalg.norm(grad - grad_o) <= 3e-2 * np.linalg.norm(grad_o)


# the device check of predict and warm_start: what was refused stays refused and
# what was accepted stays accepted, rows out of order (the host decides) and
# duplicates included
@pytest.mark.parametrize("case", ["ok", "unsorted", "duplicate", "self-loop", "one-sided", "one-sided-hub", "unsorted-one-sided"])
def test_predict_undirected_check(jc, case):
    rows = [sorted(set(jc.gen_grid(6).neighbors[o:e].tolist()))
            for o, e in zip(jc.gen_grid(6).offsets[:-1], jc.gen_grid(6).offsets[1:])]
    if case.startswith("unsorted"):
        rows[7] = rows[7][::-1]
    if case == "duplicate":
        rows[0] = [rows[0][0]] + rows[0]
    if case == "self-loop":
        rows[3] = sorted(rows[3] + [3])
    if case.endswith("one-sided"):
        rows[35] = sorted(rows[35] + [0])
    g = jc.Csr(36, np.cumsum([0] + [len(r) for r in rows]).astype(np.uint32), np.concatenate(rows).astype(np.uint32))
    if case == "one-sided-hub":
        s = star(jc, 1500, 3)
        rows = [s.neighbors[o:e].tolist() for o, e in zip(s.offsets[:-1], s.offsets[1:])]
        rows[700] = []  # the hub still lists 700
        g = jc.Csr(1501, np.cumsum([0] + [len(r) for r in rows]).astype(np.uint32), np.concatenate(rows).astype(np.uint32))
    graphs = [jc.gen_path(9), g, jc.gen_scale_free(50, 2, 1)]
    net = jc.Mpnn(2, 5)
    ev = jc.Evaluator(graphs)
    seeds = [jc.seed_uniform(x.n_nodes, 2, 3) for x in graphs]
    if case in ("ok", "unsorted", "duplicate"):
        xyz, _ = net.predict(graphs)
        assert all(np.all(np.isfinite(x)) for x in xyz)
        net.warm_start(graphs, seeds, ev)
    else:
        for call in (lambda: net.predict(graphs), lambda: net.warm_start(graphs, seeds, ev)):
            with pytest.raises(jc.JcError, match="undirected"):
                call()
        xyz, _ = net.predict(graphs[:1])  # the network stays usable
        assert np.all(np.isfinite(xyz[0]))


# pivot words of 1, 2 and blocks of 4 (and their last, partial word), several
# components, and hop distances on both sides of 65,535 (a path from its ends)
@pytest.mark.parametrize("k", [1, 63, 64, 65, 128, 129, 256, 257])
def test_multi_source_bfs_words(jc, orc, k):
    a, b = jc.gen_scale_free(700, 2, 3), jc.gen_grid(17)
    g = jc.csr_from_pairs(1000, np.concatenate([a.pairs(), b.pairs() + 700]))  # 11 isolated nodes
    e = jc.LayoutEngine("sgd-stress-gpu")
    e.set_params({"n_pivots": k, "random_pivots": True, "seed": 5})
    for _ in range(2):  # the second bind reuses the first's workspace
        e.init(g, jc.seed_uniform(1000, 2, 1))
        piv, dist = e.pivots()
        assert len(set(piv.tolist())) == k
        for t in {0, k // 2, k - 1}:
            assert np.array_equal(dist[t], orc.bfs(g, int(piv[t])))


@pytest.mark.parametrize("n", [65000, 70000])
def test_multi_source_bfs_long_path(jc, n):
    g = jc.gen_path(n)
    e = jc.LayoutEngine("sgd-stress-gpu")
    e.set_params({"n_pivots": 3, "random_pivots": True, "seed": 1})
    e.init(g, jc.seed_uniform(n, 2, 1))
    piv, dist = e.pivots()
    for t in range(3):
        assert np.array_equal(dist[t], np.abs(np.arange(n) - int(piv[t])).astype(np.uint32))


# one batch, one sample a batch, block remainders, several sweeps a step
@pytest.mark.parametrize("n,batches,sweeps", [(4096, 1, 1), (4097, 1, 2), (8192, 1, 1), (8193, 1, 1), (16384, 1, 2),
                                              (16385, 1, 2), (20000, 3, 1), (700, 700, 1), (1501, 7, 3), (33000, 0, 1)])
def test_pair_batches_bit_exact(jc, orc, n, batches, sweeps):
    g = jc.gen_watts_strogatz(n, 4, 0.2, n)
    pos = jc.seed_uniform(n, 3, 2) * np.float32(10.0)
    s = {"n_pivots": 5, "eta_max": 4.0, "sweeps_per_step": sweeps}
    e = jc.LayoutEngine("sgd-stress")
    e.set_params({**s, "scatter_batches": batches})
    e.init(g, pos)
    o = orc.Sgd(g, pos, mode=2, scatter_batches=batches, **s)
    for _ in range(3):
        assert np.array_equal(bits(e.step()), bits(o.step()))


def one_step(jc, orc, g, pos, **settings):
    e = jc.LayoutEngine("fa2-bh")
    e.set_params(settings)
    e.init(g, pos)
    e.step()
    o = orc.Fa2(g, pos, bh=True, **{k: v for k, v in settings.items() if k not in ("hub_threshold", "warp_threshold")})
    o.step()
    return e, o.get()


# attraction lists at the edges of the warp path (32 entries here, whole and
# partial chunks of 32), as the graph's size chooses it
@pytest.mark.parametrize("leaves,lin_log", [(k, False) for k in (30, 31, 32, 33, 63, 64, 65, 96, 97, 500)]
                         + [(33, True), (97, True)])
def test_attraction_list_lengths_bit_exact(jc, orc, leaves, lin_log):
    g = star(jc, leaves, leaves // 2)
    e, r = one_step(jc, orc, g, jc.seed_uniform(g.n_nodes, 3, leaves), theta=0.7, lin_log_mode=lin_log)
    f, st = e.forces()
    if lin_log:  # logf against the host's: one ulp of a term
        assert np.linalg.norm(f - r["force"]) <= 1e-6 * np.linalg.norm(r["force"])
    else:
        assert np.array_equal(bits(f), bits(r["force"])) and np.array_equal(bits(st), bits(r["stats"]))


# both sides of the walk's size rule (151,552) and of the list-length rule
# (32,768 and 196,608)
@pytest.mark.parametrize("n", [32768, 32769, 151552, 151553, 196608, 196609])
def test_walk_and_list_size_rules_bit_exact(jc, orc, n):
    g = jc.gen_scale_free(n, 2, n)
    e, r = one_step(jc, orc, g, jc.seed_uniform(n, 3, 1), theta=0.9, hub_threshold=1 << 30)
    f, _ = e.forces()
    assert np.array_equal(bits(f), bits(r["force"]))


def crowded(jc, n, far, seed):
    """A layout whose bodies share the first ten octant levels: a unit cube and
    a body at distance `far`; every third body on a coarse lattice, so keys tie
    in the high word too and whole keys repeat."""
    pos = jc.seed_uniform(n, 3, seed)
    k = np.arange(1, n, 3)
    for c in range(3):
        pos[3 * k + c] = np.round(pos[3 * k + c] * 16) / np.float32(16)
    pos[:3] = far
    return pos


# the one-launch re-sort: a single block, one block's last part, several blocks
# with barriers (2,048 bodies each), graph replays and plain launches
@pytest.mark.parametrize("use_graph", [True, False])
@pytest.mark.parametrize("n", [40, 2048, 2049, 6143, 30001])
def test_long_runs_resort_bit_exact(jc, orc, n, use_graph):
    g = jc.gen_scale_free(n, 2, n)
    pos = crowded(jc, n, 3.0e4, 5)
    e = jc.LayoutEngine("fa2-bh")
    e.set_params({"theta": 0.8, "use_graph": use_graph, "hub_threshold": 1 << 30})
    e.init(g, pos)
    o = orc.Fa2(g, pos, bh=True, theta=0.8)
    for _ in range(2):
        e.step()
        o.step()
        r = o.get()
        assert e.tree_info()["nodes"] > 0
        assert np.array_equal(bits(e.forces()[0]), bits(r["force"]))
        assert np.array_equal(bits(e.positions()), bits(r["pos"]))


def test_long_runs_resort_in_a_batch(jc):
    graphs = [jc.gen_scale_free(n, 2, n) for n in (3000, 50, 2500)]
    pos = [crowded(jc, g.n_nodes, 2.0e5, 9) for g in graphs]
    b = jc.LayoutEngine("fa2-bh")
    b.set_params({"theta": 0.8})
    b.init_batch(graphs, pos)
    out = b.step_many(3)
    at = 0
    for g, p in zip(graphs, pos):
        e = jc.LayoutEngine("fa2-bh")
        e.set_params({"theta": 0.8})
        e.init(g, p)
        assert np.array_equal(bits(out[at:at + 3 * g.n_nodes]), bits(e.step_many(3)))
        at += 3 * g.n_nodes


# both sides of the sort's tile-size rules and of the walk chain's rule
@pytest.mark.parametrize("n", [511, 512, 513, 24576, 24577, 32767, 32768, 32769, 196607, 400000, 400001])
def test_sort_tile_rules_bit_exact(jc, orc, n):
    g = jc.gen_watts_strogatz(n, 4, 0.05, n) if n < 100000 else jc.gen_path(n)
    e, r = one_step(jc, orc, g, jc.seed_uniform(n, 3, 7), theta=1.2)
    assert e.tree_info()["nodes"] == r["n_octree"]
    assert np.array_equal(bits(e.forces()[0]), bits(r["force"]))


# the warp walk: its smallest graphs, whole and partial blocks of four warps,
# both sides of its size rule (10,240) and of its theta rule (0.632), lists longer
# than one batch of 256 terms; trees past its bitmap and queues it does not hold
# (chains of close pairs, a dense ball at a small theta) go along the ropes
@pytest.mark.parametrize("case", ["n1", "n2", "n3", "n7", "n8", "n9", "n1000", "n10240", "n10241", "theta0.63", "theta0.64",
                                  "2d", "chains", "dense"])
def test_warp_walk_bit_exact(jc, orc, case):
    theta, n = 0.8, 3000
    if case[0] == "n":
        n = int(case[1:])
    if case.startswith("theta"):
        theta = float(case[5:])
    if case == "dense":
        theta, n = 0.64, 9000
    pos = jc.seed_uniform(n, 2 if case == "2d" else 3, n)
    if case == "chains":
        p = pos.reshape(n, 3)
        p[1:2001:2] = p[0:2000:2] + np.array([3e-6, -2e-6, 1e-6], np.float32)
    g = jc.gen_scale_free(n, 2, n) if n > 3 else jc.gen_path(n)
    e = jc.LayoutEngine("fa2-bh")
    e.set_params({"theta": theta})
    e.init(g, pos)
    o = orc.Fa2(g, pos, bh=True, theta=theta)
    o.set_tree_capacity(1 << 20)
    for _ in range(3):
        e.step()
        o.step()
        r = o.get()
        assert e.tree_info()["nodes"] == r["n_octree"]
        assert np.array_equal(bits(e.forces()[0]), bits(r["force"]))
        assert e.walk_counts() == (r["n_inter"], r["n_open"])


# a batch's trees built one CTA a graph: graphs around the blocks of 32, 256 and
# 1,024 bodies, each largest size on both sides of the thread and size rules (past
# 8,192 the forest's kernels), one body and none; runs of equal tops that need the
# whole key; close pairs whose chains of cells outgrow the shared lists, the ropes
# and the tree's first capacity; whole keys repeated; bodies at no position
@pytest.mark.parametrize("case", ["edges", "2048", "2049", "4096", "4097", "8192", "8193", "2d", "runs", "runs8193", "chains",
                                  "repeats", "nan", "nan8193", "many"])
def test_batch_trees_equal_single_engines(jc, case):
    big = int(case[-4:]) if case[-4:].isdigit() else 2000
    sizes = [1, 2, 3, 31, 32, 33, 255, 256, 257, 1023, 1024, 1025] if case == "edges" else [50, big, 1, 700, min(big, 2000)]
    if case == "many":  # more bodies than the walk's size rule (151,552)
        sizes = [8000 - k for k in range(20)]
    graphs = [jc.gen_scale_free(n, 2, n) if n > 3 else jc.gen_path(n) for n in sizes]
    pos = [jc.seed_uniform(n, 2 if case == "2d" else 3, 3 * n) for n in sizes]
    if case.startswith("runs"):
        pos = [crowded(jc, n, 3.0e4, 11) if n > 40 else p for n, p in zip(sizes, pos)]
    for n, p in zip(sizes, pos):
        p = p.reshape(n, 3)
        if case == "chains" and n > 40:
            p[1:n - 1:2] = p[0:n - 2:2] + np.array([3e-6, -2e-6, 1e-6], np.float32)
        if case == "repeats" and n > 40:
            p[40:80 if n > 80 else n] = p[:min(n, 80) - 40]
        if case.startswith("nan"):
            p[0 if n < 40 else 7, 1] = np.nan
    b = jc.LayoutEngine("fa2-bh")
    b.set_params({"theta": 0.8})
    b.init_batch(graphs, pos)
    es = []
    for g, p in zip(graphs, pos):
        e = jc.LayoutEngine("fa2-bh")
        e.set_params({"theta": 0.8, "hub_threshold": 1 << 30, "warp_threshold": 1 << 30})
        e.init(g, p)
        es.append(e)
    for _ in range(3):
        b.step_many(1)
        for e in es:
            e.step_many(1)
        for x, y in ((b.forces()[0], [e.forces()[0] for e in es]), (b.positions(), [e.positions() for e in es])):
            y = np.concatenate(y)
            assert np.array_equal(np.isnan(x), np.isnan(y))
            assert np.array_equal(bits(x)[~np.isnan(x)], bits(y)[~np.isnan(y)])
        assert b.tree_info()["nodes"] == sum(e.tree_info()["nodes"] for e in es)
        assert b.walk_counts() == tuple(sum(c) for c in zip(*(e.walk_counts() for e in es)))


# a single graph's tree in one launch: both sides of its thread and size rules
# (256, 3,072), the rope walks on its tree, bodies at no position and whole keys
# repeated
@pytest.mark.parametrize("case", ["256", "257", "1024", "1025", "3072", "3073", "rope", "nan", "repeats"])
def test_single_graph_trees_bit_exact(jc, orc, case):
    n = int(case) if case.isdigit() else 500
    pos = jc.seed_uniform(n, 3, n)
    p = pos.reshape(n, 3)
    if case == "nan":
        p[[3, 499], 1] = np.nan
    if case == "repeats":
        p[40:80] = p[:40]
    g = jc.gen_scale_free(n, 2, n)
    theta = 0.5 if case == "rope" else 0.8
    e = jc.LayoutEngine("fa2-bh")
    e.set_params({"theta": theta})
    e.init(g, pos)
    e.step()
    o = orc.Fa2(g, pos, bh=True, theta=theta)
    o.set_tree_capacity(1 << 20)  # repeated keys reach the depth cap
    o.step()
    r = o.get()
    assert e.tree_info()["nodes"] == r["n_octree"]
    f, _ = e.forces()
    nan = np.isnan(r["force"])
    assert np.array_equal(np.isnan(f), nan)
    assert np.array_equal(bits(f)[~nan], bits(r["force"])[~nan])
    assert e.walk_counts() == (r["n_inter"], r["n_open"])


# the no-allocation pass: rows around the 32 entries a warp takes together (whole
# and partial chunks), 40 such rows in two warps, row orders of whole and partial
# warps, one body, both sides of the tree's size rule (3,072)
@pytest.mark.parametrize("case", ["star31", "star32", "star33", "star64", "star97", "clique40", "1", "2", "31", "32", "33",
                                  "3072", "3073"])
def test_noalloc_rows_bit_exact(jc, orc, case):
    torch = pytest.importorskip("torch")
    if case.startswith("star"):
        g = star(jc, int(case[4:]), int(case[4:]))
    elif case == "clique40":
        g = jc.csr_from_pairs(40, np.array([(a, b) for a in range(40) for b in range(a + 1, 40)], np.uint32))
    else:
        g = jc.gen_scale_free(int(case), 2, 3) if int(case) > 3 else jc.gen_path(int(case))
    pos = jc.seed_uniform(g.n_nodes, 3, 21)
    off, nbr = (torch.from_numpy(a.view(np.int32).copy()).cuda() for a in (g.offsets, g.neighbors))
    p, out = torch.from_numpy(pos).cuda(), torch.full((3 * g.n_nodes,), float("nan"), device="cuda")
    torch.cuda.synchronize()
    for _ in range(2):
        jc.fa2_bh_forces_noalloc(g.n_nodes, off.data_ptr(), nbr.data_ptr(), p.data_ptr(), out.data_ptr(), theta=0.7)
        o = orc.Fa2(g, pos, bh=True, theta=0.7)
        o.step()
        assert np.array_equal(bits(out.cpu().numpy()), bits(o.get()["force"]))


# graphs of no bodies in a batch, on both of its tree paths
@pytest.mark.parametrize("big", [300, 8193])
def test_empty_graphs_in_a_batch(jc, big):
    none = jc.Csr(0, np.zeros(1, np.uint32), np.zeros(0, np.uint32))
    g = [jc.gen_scale_free(big, 2, 1), jc.gen_scale_free(40, 2, 2)]
    p = [jc.seed_uniform(big, 3, 3), jc.seed_uniform(40, 3, 4)]
    b = jc.LayoutEngine("fa2-bh")
    b.init_batch([none, g[0], none, g[1], none], [np.zeros(0, np.float32), p[0], np.zeros(0, np.float32), p[1],
                                                  np.zeros(0, np.float32)])
    out = b.step_many(3)
    alone = []
    for x, y in zip(g, p):
        e = jc.LayoutEngine("fa2-bh")
        e.init(x, y)
        alone.append(e.step_many(3))
    assert np.array_equal(bits(out), bits(np.concatenate(alone)))
