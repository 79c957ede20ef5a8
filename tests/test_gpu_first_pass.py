"""Whether a run builds the index of its graph depends on its steps: walks
without an index, through sample levels and through membership tables are the
same, in the order in which a handle comes to them."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("algo,p,q,weighted", [(0, 0.5, 2.0, False), (0, 0.25, 4.0, False), (1, 0.5, 2.0, False),
                                               (0, 2.0, 0.5, True)])
@pytest.mark.parametrize("device", [False, True])
def test_short_runs_then_long_ones(gw, oracle, algo, p, q, weighted, device):
    """A few walkers (no index), all of them (tables), a few again, a new graph."""
    import torch
    for seed in (1, 2):
        beg, csr = oracle.rmat_graph(13, seed=seed)
        V, term = len(beg) - 1, 0.15 if algo else 0.0
        w = np.random.default_rng(seed).lognormal(0.0, 1.0, len(csr)).astype(np.float32) if weighted else None
        alias = oracle.build_alias(beg, w) if weighted else None
        if seed == 1:
            eng = gw.WalkEngine(algorithm=algo, maxhops=20, p=p, q=q, alpha=0.2, term_prob=term, seed=3)
        if device:
            d = [torch.from_numpy(beg.view(np.int64)).cuda(), torch.from_numpy(csr.view(np.int32)).cuda()]
            eng.set_device_graph(V, len(csr), d[0].data_ptr(), d[1].data_ptr())
            if weighted:
                d.append(torch.from_numpy(w).cuda())
                eng.set_device_weights(d[2].data_ptr())
        else:
            eng.set_host_graph(beg, csr)
            if weighted:
                eng.set_host_weights(w)
        cfg = oracle.make_cfg(algo=algo, maxhops=20, p=p, q=q, alpha=0.2, term_prob=term, seed=3, wps=8)
        for first, count in ((V, 300), (0, 8 * V), (5 * V, 1), (7, 2 * V)):
            eng.init_walkers(algo, 8, 3, first=first, count=count)
            st = eng.run()
            ref = oracle.walk(beg, csr, cfg, first, count, paths=False, alias=alias)
            assert np.array_equal(eng.hashes(), ref["hashes"])
            assert (st["steps"], st["trials"]) == (ref["stats"]["steps"], ref["stats"]["trials"])
    eng.close()


@pytest.mark.parametrize("p,q", [(2.0, 0.5), (0.25, 4.0)])
def test_levels_walk_as_tables(gw, oracle, p, q):
    """A CSR that the L2 does not keep: its first run reads sample levels, a run of few
    walkers none, a later one tables; the first's hashes against theirs, and
    against the oracle's for some walkers."""
    dg = gw.DeviceGraph(21, nverts=2_000_003, edgefactor=12, seed=5, symmetric=True)
    assert 4 * dg.nedges > 126 << 20
    beg, csr = dg.to_host()
    eng = gw.WalkEngine(algorithm=0, maxhops=10, p=p, q=q, seed=4)
    eng.set_device_graph(dg.nverts, dg.nedges, dg.beg_ptr, dg.csr_ptr)
    eng.init_walkers()
    eng.run()
    levels = eng.hashes()
    cfg = oracle.make_cfg(algo=0, maxhops=10, p=p, q=q, seed=4)
    at = int(np.searchsorted(beg, dg.nedges // 2)) - 1500
    for first in (0, at):
        assert np.array_equal(levels[first:first + 3000],
                              oracle.walk(beg, csr, cfg, first, 3000, paths=False)["hashes"])
    eng.init_walkers(0, 1, 4, first=at, count=5000)
    eng.run()
    assert np.array_equal(eng.hashes(), levels[at:at + 5000])
    eng.set_config(maxhops=200)
    eng.init_walkers()
    eng.run()  # 200 hops of 2 M walkers: tables
    eng.set_config(maxhops=10)
    eng.init_walkers()
    eng.run()
    assert np.array_equal(eng.hashes(), levels)
    eng.close()
    dg.free()


def test_levels_where_tables_find_no_room(gw, oracle):
    """23 M edges: the memory of tables (252 MB) is asked for ahead, and refused;
    the levels (3 MB) that the run reads have room."""
    import torch
    dg = gw.DeviceGraph(19, nverts=1 << 19, edgefactor=24, nsamples=24 << 19, seed=3, symmetric=True)
    assert 6 * dg.nedges > 126 << 20 and 10 * dg.nedges + 48 * dg.nverts < 256 << 20
    beg, csr = dg.to_host()
    eng = gw.WalkEngine(algorithm=0, maxhops=6, p=2.0, q=0.5, seed=4)
    eng.set_device_graph(dg.nverts, dg.nedges, dg.beg_ptr, dg.csr_ptr)
    eng.init_walkers()
    torch.cuda.empty_cache()
    fill = torch.empty(torch.cuda.mem_get_info()[0] - (100 << 20), dtype=torch.uint8, device="cuda")
    eng.run()
    got = eng.hashes()[:4000]
    del fill
    torch.cuda.empty_cache()
    ref = oracle.walk(beg, csr, oracle.make_cfg(algo=0, maxhops=6, p=2.0, q=0.5, seed=4), 0, 4000, paths=False)
    assert np.array_equal(got, ref["hashes"])
    eng.run()
    assert np.array_equal(eng.hashes()[:4000], ref["hashes"])
    eng.close()
    dg.free()
