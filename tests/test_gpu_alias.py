"""Alias tables of hub vertices (built a window at a time): one-step weighted
walks from hubs whose degrees sit around the windows' size equal the oracle's,
for weights that fill the two queues in every proportion."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

DEGREES = [257, 1023, 1024, 1025, 2047, 2048, 2049, 3000, 5000, 20000]


def weights_of(kind, n, rng):
    if kind == "one_large":  # one column takes from all others
        w = np.full(n, 0.5)
        w[rng.integers(0, n)] = 10.0 * n
    elif kind == "one_small":
        w = np.full(n, 1.0)
        w[rng.integers(0, n)] = 1e-3
    elif kind == "larges_last":  # every small is consumed before any dropped large
        w = np.where(np.arange(n) < n // 2, 0.25, 1.75)
    elif kind == "pareto":
        w = rng.pareto(1.2, n) + 1e-4
    elif kind == "equal":
        w = np.full(n, 3.0)
    else:
        w = rng.lognormal(0, 1, n)
    return w.astype(np.float32)


@pytest.mark.parametrize("kind", ["one_large", "one_small", "larges_last", "pareto", "equal", "lognormal"])
def test_hub_alias_tables_match_oracle(gw, oracle, kind):
    rng = np.random.default_rng(4)
    V = 1024
    degrees = np.zeros(V, np.int64)
    degrees[:len(DEGREES)] = DEGREES
    beg = np.zeros(V + 1, np.uint64)
    beg[1:] = np.cumsum(degrees)
    # neighbours spread over the ids, so that a wrong column shows
    csr = np.concatenate([np.sort(rng.integers(0, V, d)) for d in degrees]).astype(np.uint32)
    w = np.concatenate([weights_of(kind, d, rng) for d in DEGREES])
    wps = 1500
    eng = gw.WalkEngine(algorithm=0, maxhops=1, p=1.0, q=1.0, seed=21, walkpersource=wps)
    eng.set_host_graph(beg, csr)
    eng.set_host_weights(w)
    eng.init_walkers(0, wps, 21, first=0, count=len(DEGREES) * wps)
    eng.run()
    ref = oracle.walk(beg, csr, oracle.make_cfg(algo=0, maxhops=1, p=1.0, q=1.0, seed=21, wps=wps), 0,
                      len(DEGREES) * wps, paths=False, alias=oracle.build_alias(beg, w))
    assert np.array_equal(eng.hashes(), ref["hashes"])
    eng.close()
