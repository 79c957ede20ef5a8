"""A call that runs out of device memory is refused and leaves the handle
usable: the outputs and the out-of-core walkers of a population that did not
fit are not taken for those of a later, smaller one."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

NOMEM, STATE = -3, -4  # GW_ERR_NOMEM, GW_ERR_STATE


def graph(oracle):
    src, dst = oracle.rmat_edges(12, 0, 8 << 12, seed=4)
    keep = (src < 2000) & (dst < 2000)
    return oracle.build_csr(2000, src[keep], dst[keep], symmetric=True)


def refused(gw, status, call):
    with pytest.raises(gw.GwError) as e:
        call()
    assert e.value.status == status


def check(eng, oracle, beg, csr, wps, maxhops):
    ref = oracle.walk(beg, csr, oracle.make_cfg(algo=0, maxhops=maxhops, p=0.5, q=2.0, seed=5, wps=wps), 0,
                      wps * (len(beg) - 1), paths=True)
    P, L = eng.paths()
    assert np.array_equal(eng.hashes(), ref["hashes"])
    assert np.array_equal(L, ref["lens"]) and np.array_equal(P, ref["paths"])


def test_paths_that_do_not_fit(gw, oracle):
    """4 TB of paths (1 M walkers of 1 M hops) after a population that fits, then a smaller one."""
    beg, csr = graph(oracle)
    eng = gw.WalkEngine(algorithm=0, maxhops=10, p=0.5, q=2.0, seed=5, record_paths=1)
    eng.set_host_graph(beg, csr)
    eng.init_walkers(0, 8, 5)
    eng.run()
    eng.set_config(maxhops=999_999)
    refused(gw, NOMEM, lambda: eng.init_walkers(0, 500, 5))
    refused(gw, STATE, eng.run)
    assert eng.num_walkers() == 0
    eng.set_config(maxhops=10)
    eng.init_walkers(0, 2, 5)
    eng.run()
    check(eng, oracle, beg, csr, 2, 10)
    eng.close()


def test_out_of_core_walkers_that_do_not_fit(gw, oracle):
    """4.2 G walkers have room for their 50 GB of hashes and lengths, not for
    the 200 GB of their records and order; the earlier population's size then
    walks again."""
    from gowalker_b200.preprocess import split_equal_edge_mass
    beg, csr = graph(oracle)
    vb, eb = split_equal_edge_mass(beg, 8)
    cache = len(beg) * 8 + 4 * ((int(np.diff(eb.astype(np.int64)).max()) + 3) & ~3) * 4
    eng = gw.WalkEngine(algorithm=0, maxhops=10, p=0.5, q=2.0, seed=5, cache_size=cache)
    eng.set_host_graph(beg, csr, vb, eb)
    eng.init_walkers(0, 4, 5)
    eng.run()
    eng.init_walkers(0, 2_100_000, 5)
    refused(gw, NOMEM, eng.run)
    eng.init_walkers(0, 4, 5)
    eng.set_config(record_paths=1)
    eng.init_walkers(0, 4, 5)
    eng.run()
    check(eng, oracle, beg, csr, 4, 10)
    eng.close()
