"""Faults that were found in use, each held by the smallest call that shows it."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def bits(a):
    return np.ascontiguousarray(a, dtype=np.float32).view(np.uint32)


def _concurrently(calls):
    """Runs each call in a thread of its own; the exceptions they raised."""
    errors = []
    gate = threading.Barrier(len(calls))

    def go(f):
        gate.wait()
        try:
            f()
        except Exception as e:  # noqa: BLE001
            errors.append(e)

    ts = [threading.Thread(target=go, args=(f,)) for f in calls]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    return errors


# Engines on two threads launch one kernel with different amounts of shared memory:
# batches whose largest graphs differ, and stress engines of different pivot counts.
# (New settings make the next step capture and instantiate its graph anew.)
@pytest.mark.parametrize("kind", ["batch", "stress"])
def test_shared_memory_limit_is_no_engines_own(jc, kind):
    def work(big, pivots):
        if kind == "batch":
            graphs = [jc.gen_scale_free(n, 2, n) for n in (big, 60)]
            e = jc.LayoutEngine("fa2-bh")
            e.init_batch(graphs, [jc.seed_uniform(g.n_nodes, 2, 1) for g in graphs])
            settings = [{"gravity": 1.0}, {"gravity": 2.0}]
        else:
            g = jc.gen_grid(90)
            e = jc.LayoutEngine("sgd-stress-gpu")
            e.set_params({"n_pivots": pivots, "random_pivots": True})
            e.init(g, jc.seed_uniform(g.n_nodes, 2, 1) * np.float32(90))
            settings = [{"n_pivots": pivots, "random_pivots": True, "sweeps_per_step": k} for k in (1, 2)]

        def go():
            for k in range(200):
                e.set_params(settings[k % 2])
                e.step_many(1, readback=False)

        return go

    assert _concurrently([work(8000, 6000), work(4200, 3500)]) == []
