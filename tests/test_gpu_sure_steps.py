"""Walks whose every trial accepts (p = q = 1), where test_gpu_first_order.py does
not go: weighted ones over many hops, one walker alone, after a run that built
the graph's tables, and through gw_walk_noalloc."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("count", [1, 2, 31, 5000, 200_000])
@pytest.mark.parametrize("tables", [False, True])
@pytest.mark.parametrize("device", [False, True])
def test_weighted_sure_steps_match_oracle(gw, oracle, count, tables, device):
    import torch
    beg, csr = oracle.rmat_graph(13, seed=4)
    V = len(beg) - 1
    w = np.random.default_rng(6).lognormal(0.0, 1.0, len(csr)).astype(np.float32)
    eng = gw.WalkEngine(algorithm=0, maxhops=25, p=0.5, q=2.0, seed=10, walkpersource=32, record_paths=1)
    if device:
        d = [torch.from_numpy(x).cuda() for x in (beg.view(np.int64), csr.view(np.int32), w)]
        eng.set_device_graph(V, len(csr), d[0].data_ptr(), d[1].data_ptr())
        eng.set_device_weights(d[2].data_ptr())
    else:
        eng.set_host_graph(beg, csr)
        eng.set_host_weights(w)
    if tables:
        eng.init_walkers()
        eng.run()
    eng.set_config(p=1.0, q=1.0)
    first = 32 * 11
    eng.init_walkers(first=first, count=count)
    st = eng.run()
    ref = oracle.walk(beg, csr, oracle.make_cfg(algo=0, maxhops=25, p=1.0, q=1.0, seed=10, wps=32), first, count,
                      paths=True, alias=oracle.build_alias(beg, w))
    P, L = eng.paths()
    assert np.array_equal(L, ref["lens"]) and np.array_equal(P, ref["paths"])
    assert np.array_equal(eng.hashes(), ref["hashes"])
    assert (st["steps"], st["trials"]) == (ref["stats"]["steps"], ref["stats"]["trials"])
    eng.close()


@pytest.mark.parametrize("nverts,numwalks", [(4096, 1), (4096, 777), (4096, 200_000)])
def test_sure_steps_without_allocation(gw, oracle, nverts, numwalks):
    import torch
    beg, csr = oracle.rmat_graph(12, seed=4)
    d_beg, d_csr = torch.from_numpy(beg.view(np.int64)).cuda(), torch.from_numpy(csr.view(np.int32)).cuda()
    cfg = gw.default_config(algorithm=0, maxhops=18, p=1.0, q=1.0, seed=3, init_mode=2, numwalks=numwalks,
                            record_paths=1)
    hashes = torch.empty(numwalks, dtype=torch.int64, device="cuda")
    lens = torch.empty(numwalks, dtype=torch.int32, device="cuda")
    paths = torch.empty((numwalks, 19), dtype=torch.int32, device="cuda")
    p = [ctypes.c_void_p(t.data_ptr()) for t in (d_beg, d_csr, hashes, lens, paths)]
    torch.cuda.synchronize()
    rc = gw.load().gw_walk_noalloc(ctypes.byref(cfg), p[0], p[1], nverts, len(csr), numwalks, p[2], p[3], p[4], None, None)
    assert rc == 0
    ref = oracle.walk(beg, csr, oracle.make_cfg(algo=0, maxhops=18, p=1.0, q=1.0, seed=3, init_mode=2,
                                                numwalks=numwalks), 0, numwalks, paths=True)
    assert np.array_equal(hashes.cpu().numpy().view(np.uint64), ref["hashes"])
    assert np.array_equal(lens.cpu().numpy().view(np.uint32), ref["lens"])
    assert np.array_equal(paths.cpu().numpy().view(np.uint32), ref["paths"])
