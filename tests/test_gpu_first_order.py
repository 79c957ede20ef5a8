"""Walks whose every trial accepts (p = q = 1) equal the oracle's: one walker,
a few, a wave and more than a wave of them, weighted and unweighted, with paths
and dead ends."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nverts,scale,wps,paths", [(3, 4, 1, 1), (1939, 11, 2, 1), (60_001, 16, 4, 1),
                                                    (262_144, 18, 4, 0)])
@pytest.mark.parametrize("symmetric", [True, False])
def test_sure_steps_match_oracle(gw, oracle, nverts, scale, wps, paths, symmetric):
    dg = gw.DeviceGraph(scale, nverts=nverts, edgefactor=16, seed=3, symmetric=symmetric)
    beg, csr = dg.to_host()
    eng = gw.WalkEngine(algorithm=0, maxhops=12, p=1.0, q=1.0, seed=8, walkpersource=wps,
                        record_paths=gw.GW_PATHS_FULL if paths else gw.GW_PATHS_NONE)
    eng.set_host_graph(beg, csr)
    eng.init_walkers(0, wps, 8)
    st = eng.run()
    ref = oracle.walk(beg, csr, oracle.make_cfg(algo=0, maxhops=12, p=1.0, q=1.0, seed=8, wps=wps), 0, wps * nverts,
                      paths=bool(paths))
    assert np.array_equal(eng.hashes(), ref["hashes"])
    assert (st["steps"], st["trials"]) == (ref["stats"]["steps"], ref["stats"]["trials"])
    eng.close()
