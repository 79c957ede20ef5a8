"""Times that an out-of-core run reports: the step kernels' own, whatever the
compute stream waits for behind them."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_step_time_without_the_wait_for_a_decision(gw):
    """The annealed choice over 60 blocks takes some hundred times a step of 2,000
    walkers; with prefetch it runs beside the step, and the re-bucketing waits
    for it.  A step takes the same with prefetch and without, three times as
    long at most (one step's walkers differ, by less)."""
    from gowalker_b200.preprocess import split_equal_edge_mass
    dg = gw.DeviceGraph(15, nverts=30_000, edgefactor=16, seed=3, symmetric=True)
    beg, csr = dg.to_host()
    dg.free()
    vb, eb = split_equal_edge_mass(beg, 60)
    cache = len(beg) * 8 + 30 * (int(np.diff(eb.astype(np.int64)).max()) + 4) * 4
    per_step = []
    for prefetch in (0, 1):
        eng = gw.WalkEngine(algorithm=0, maxhops=20, p=0.5, q=2.0, seed=5, cache_size=cache, prefetch=prefetch,
                            init_mode=2, numwalks=2000)
        eng.set_host_graph(beg, csr, vb, eb)
        for _ in range(2):
            eng.init_walkers()
            st = eng.run(2)  # GW_POLICY_SA
        assert 0 < st["kernel_ms"] + st["bucket_ms"] < st["total_ms"]
        per_step.append(st["kernel_ms"] / st["iterations"])
        eng.close()
    assert per_step[1] < 3 * per_step[0]
