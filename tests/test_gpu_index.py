"""The index of a resident CSR (vertex records, membership tables): walks that
search N(prev) on most trials equal the oracle's on graphs whose degrees sit
around a bucket's size, with repeated neighbours, hubs, isolated vertices, and
on a borrowed CSR that starts at any word."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def graph_of(degrees, repeat, rng):
    """Sorted random neighbour lists of the given degrees, each id `repeat` times."""
    V = len(degrees)
    lists = [np.sort(np.repeat(rng.integers(0, V, -(-d // repeat)), repeat)[:d]) for d in degrees]
    beg = np.zeros(V + 1, np.uint64)
    beg[1:] = np.cumsum([len(x) for x in lists])
    return beg, np.concatenate(lists + [np.zeros(0, np.int64)]).astype(np.uint32)


@pytest.mark.parametrize("name,repeat", [("edges_of_buckets", 1), ("repeats", 9), ("hub", 1), ("sparse", 1)])
@pytest.mark.parametrize("algo", [0, 1])
def test_index_walks_match_oracle(gw, oracle, name, repeat, algo):
    rng = np.random.default_rng(5)
    degrees = {
        "edges_of_buckets": list(range(1, 70)) * 20 + [0, 255, 256, 257, 1000],
        "repeats": rng.integers(1, 90, 700).tolist(),
        "hub": [50000, 1, 2] + rng.integers(0, 12, 4000).tolist(),
        "sparse": ([0] * 97 + [3]) * 60,
    }[name]
    beg, csr = graph_of(degrees, repeat, rng)
    V = len(degrees)
    term = 0.15 if algo else 0.0
    eng = gw.WalkEngine(algorithm=algo, maxhops=25, p=0.5, q=2.0, alpha=0.2, term_prob=term, seed=9, walkpersource=2)
    eng.set_host_graph(beg, csr)
    eng.init_walkers(algo, 2, 9)
    st = eng.run()
    cfg = oracle.make_cfg(algo=algo, maxhops=25, p=0.5, q=2.0, alpha=0.2, term_prob=term, seed=9, wps=2)
    ref = oracle.walk(beg, csr, cfg, 0, 2 * V, paths=False)
    assert np.array_equal(eng.hashes(), ref["hashes"])
    assert (st["steps"], st["trials"]) == (ref["stats"]["steps"], ref["stats"]["trials"])
    eng.close()


@pytest.mark.parametrize("algo,offset", [(0, 0), (0, 1), (1, 3), (0, 8)])
def test_walks_on_borrowed_csr_at_any_word(gw, oracle, algo, offset):
    import torch
    beg, csr = oracle.rmat_graph(12, 16, seed=6)
    V = len(beg) - 1
    d_beg = torch.from_numpy(beg.view(np.int64)).cuda()
    d_csr = torch.zeros(len(csr) + 16, dtype=torch.int32, device="cuda")
    d_csr[offset:offset + len(csr)] = torch.from_numpy(csr.view(np.int32)).cuda()
    term = 0.15 if algo else 0.0
    eng = gw.WalkEngine(algorithm=algo, maxhops=30, p=0.5, q=2.0, alpha=0.2, term_prob=term, seed=3)
    eng.set_device_graph(V, len(csr), d_beg.data_ptr(), d_csr.data_ptr() + 4 * offset)
    eng.init_walkers(algo, 1, 3)
    eng.run()
    cfg = oracle.make_cfg(algo=algo, maxhops=30, p=0.5, q=2.0, alpha=0.2, term_prob=term, seed=3)
    assert np.array_equal(eng.hashes(), oracle.walk(beg, csr, cfg, 0, V, paths=False)["hashes"])
    eng.close()


def test_index_gives_way_to_outputs(gw, oracle):
    """With the device full, a population whose outputs fit only in the memory
    of the index still walks, without it."""
    import torch
    dg = gw.DeviceGraph(18, nverts=1 << 18, edgefactor=16, seed=7, symmetric=True)
    beg, csr = dg.to_host()
    eng = gw.WalkEngine(algorithm=0, maxhops=4, p=0.5, q=2.0, seed=5)
    eng.set_device_graph(dg.nverts, dg.nedges, dg.beg_ptr, dg.csr_ptr)
    eng.init_walkers(0, 1, 5)
    eng.run()  # builds the index: some 90 MB
    torch.cuda.empty_cache()
    fill = torch.empty(torch.cuda.mem_get_info()[0] - (60 << 20), dtype=torch.uint8, device="cuda")
    eng.init_walkers(0, 32, 5)  # 12 bytes for each of 8.4 M walkers: 101 MB
    eng.run()
    got = eng.hashes()[:2000]
    del fill
    torch.cuda.empty_cache()
    ref = oracle.walk(beg, csr, oracle.make_cfg(algo=0, maxhops=4, p=0.5, q=2.0, seed=5, wps=32), 0, 2000, paths=False)
    assert np.array_equal(got, ref["hashes"])
    eng.close()
