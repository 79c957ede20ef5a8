"""The index of a resident graph gives way to what else needs the memory: other
engines, edge lists, the out-of-core state of the same engine, the next graph;
a later run builds it again where there is room."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

MB = 1 << 20


def filled(leave):
    """All of the device's memory but `leave` bytes."""
    import torch
    torch.cuda.empty_cache()
    return torch.empty(torch.cuda.mem_get_info()[0] - leave, dtype=torch.uint8, device="cuda")


@pytest.fixture
def indexed(gw, oracle):
    """An engine that keeps an index of 90 MB, and its walks."""
    dg = gw.DeviceGraph(18, nverts=1 << 18, edgefactor=16, seed=7, symmetric=True)
    beg, csr = dg.to_host()
    eng = gw.WalkEngine(algorithm=0, maxhops=40, p=0.5, q=2.0, seed=5)
    eng.set_device_graph(dg.nverts, dg.nedges, dg.beg_ptr, dg.csr_ptr)
    eng.init_walkers()
    eng.run()
    ref = oracle.walk(beg, csr, oracle.make_cfg(algo=0, maxhops=40, p=0.5, q=2.0, seed=5), 0, 2000, paths=False)
    assert np.array_equal(eng.hashes()[:2000], ref["hashes"])
    yield eng, eng.hashes(), beg, csr
    eng.close()
    dg.free()


def again(eng, hashes):
    for _ in range(2):
        eng.init_walkers()
        eng.run()
        assert np.array_equal(eng.hashes(), hashes)


def test_to_another_engine(gw, indexed):
    eng, hashes, beg, csr = indexed
    fill = filled(60 * MB)
    other = gw.WalkEngine(algorithm=0, maxhops=4, p=0.5, q=2.0, seed=5)
    small = np.arange(1001, dtype=np.uint64)
    other.set_host_graph(small, np.arange(1000, dtype=np.uint32)[::-1].copy())
    other.init_walkers(0, 8400, 5)  # 12 bytes for each of 8.4 M walkers: 101 MB
    assert other.run()["walkers"] == 8_400_000
    other.close()
    del fill
    import torch
    torch.cuda.empty_cache()
    again(eng, hashes)


def test_to_an_edge_list(gw, indexed):
    import torch
    eng, hashes, beg, csr = indexed
    n = 5_000_000
    src = torch.arange(n, dtype=torch.int32, device="cuda") % 70001
    dst = (src + 1 + torch.arange(n, dtype=torch.int32, device="cuda") // 70001) % 70001
    fill = filled(60 * MB)
    g = gw.DeviceGraph.from_edges(src, dst, nverts=70001)  # 16 bytes of keys a pair: 80 MB
    assert g.nedges == n
    g.free()
    del fill, src, dst
    torch.cuda.empty_cache()
    again(eng, hashes)


def test_to_its_own_out_of_core_run(gw, oracle):
    """Two blocks of 3.8 M edges, weighted: the slots find room, the alias
    tables' scratch (28 bytes an edge of a block) only where the index was."""
    import torch
    from gowalker_b200.preprocess import split_equal_edge_mass
    dg = gw.DeviceGraph(18, nverts=1 << 18, edgefactor=16, seed=7, symmetric=True)
    beg, csr = dg.to_host()
    dg.free()
    vb, eb = split_equal_edge_mass(beg, 2)
    w = np.random.default_rng(1).lognormal(0, 1, len(csr)).astype(np.float32)
    eng = gw.WalkEngine(algorithm=0, maxhops=40, p=0.5, q=2.0, seed=5, cache_size=1 << 34)
    eng.set_host_graph(beg, csr, vb, eb)
    eng.init_walkers()
    eng.run()  # in core: the index
    eng.set_host_weights(w)
    maxe = int(np.diff(eb.astype(np.int64)).max())
    slots = 2 * 12 * (maxe + 4)
    eng.set_config(cache_size=len(beg) * 8 + slots)
    eng.init_walkers()
    fill = filled(slots + len(beg) * 8 + 60 * MB)
    eng.run()
    del fill
    torch.cuda.empty_cache()
    ref = oracle.walk(beg, csr, oracle.make_cfg(algo=0, maxhops=40, p=0.5, q=2.0, seed=5), 0, 2000, paths=False,
                      alias=oracle.build_alias(beg, w))
    assert np.array_equal(eng.hashes()[:2000], ref["hashes"])
    eng.close()


def test_to_the_next_graph(gw):
    """The index of 31 M edges, 340 MB, goes when a smaller graph comes."""
    import torch
    dg = gw.DeviceGraph(20, nverts=1 << 20, edgefactor=16, seed=7, symmetric=True)
    eng = gw.WalkEngine(algorithm=0, maxhops=240, p=0.5, q=2.0, seed=5)  # eight steps an edge: tables
    eng.set_device_graph(dg.nverts, dg.nedges, dg.beg_ptr, dg.csr_ptr)
    eng.init_walkers()
    before = torch.cuda.mem_get_info()[0]
    eng.run()
    with_index = torch.cuda.mem_get_info()[0]
    assert before - with_index > 300 * MB
    eng.set_host_graph(np.arange(1001, dtype=np.uint64), np.arange(1000, dtype=np.uint32)[::-1].copy())
    assert torch.cuda.mem_get_info()[0] - with_index > 300 * MB
    eng.close()
    dg.free()
