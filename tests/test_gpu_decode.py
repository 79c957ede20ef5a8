"""Compressed blocks decoded by id ranges: out-of-core walks equal the oracle's
on blocks whose vertices sit around a chunk, a task and a split group, with
long runs of vertices without neighbours between and behind them, and with
hubs among small vertices."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

DEGREES = {
    "chunk_edges": [31, 32, 33, 63, 64, 65, 1, 0, 2] * 60,
    "task_edges": [127, 128, 129, 1023, 1024, 1025, 1, 3] * 12,
    "empty_runs": ([150] * 8 + [0] * 200) * 10 + [900] + [0] * 700 + [2, 0, 0, 40] + [0] * 300,
    "hubs": ([1, 2, 3, 4000, 1, 0, 1100, 2] + [1] * 40) * 8,
    "one_vertex_blocks": [2000] * 8,
}


@pytest.mark.parametrize("prefetch", [0, 1])
@pytest.mark.parametrize("name", sorted(DEGREES))
def test_decoded_blocks_walk_like_oracle(gw, oracle, name, prefetch):
    rng = np.random.default_rng(len(name))
    degrees = np.array(DEGREES[name])
    V = max(len(degrees), 8)
    lists = [np.sort(rng.integers(0, V, d)) for d in degrees]
    beg = np.zeros(V + 1, np.uint64)
    beg[1:] = np.cumsum(degrees)
    csr = np.concatenate(lists).astype(np.uint32)
    vb, eb = oracle.split_equal_edge_mass(beg, 8)
    slot = ((int(np.diff(eb.astype(np.int64)).max()) + 3) & ~3) * 4
    # the vertex offsets, one staging buffer per upload in flight (a block
    # compresses to no more than its ids and its vertices' offsets, two bytes a
    # chunk and twelve a split group), and three slots
    stage = slot + slot // 8 + 4 * int(np.diff(vb.astype(np.int64)).max()) + 512
    cache = (V + 1) * 8 + (1 + prefetch) * stage + 3 * slot
    assert cache < (V + 1) * 8 + 4 * len(csr)
    eng = gw.WalkEngine(algorithm=0, maxhops=20, p=0.5, q=2.0, seed=12, walkpersource=3, compress_blocks=1,
                        prefetch=prefetch, cache_size=cache)
    eng.set_host_graph(beg, csr, vb, eb)
    eng.init_walkers(0, 3, 12)
    st = eng.run()
    ref = oracle.walk(beg, csr, oracle.make_cfg(algo=0, maxhops=20, p=0.5, q=2.0, seed=12, wps=3), 0, 3 * V,
                      paths=False)
    assert st["block_loads"] > 0
    assert np.array_equal(eng.hashes(), ref["hashes"])
    eng.close()


@pytest.mark.parametrize("prefetch", [0, 1])
def test_blocks_of_one_to_four_pieces(gw, oracle, prefetch):
    """A prefetched block arrives in one to four pieces by its payload (2 MB
    each at least): blocks of 0.5 to 4.5 M ids, about 2 bytes an id."""
    rng = np.random.default_rng(3)
    deg = 64
    sizes = [4_500_000, 500_000, 2_200_000, 3_200_000, 1_200_000] * 2
    vb = np.concatenate([[0], np.cumsum([n // deg for n in sizes])]).astype(np.uint32)
    V = int(vb[-1])
    csr = np.sort(rng.integers(0, V, (V, deg), dtype=np.uint32), axis=1).ravel()
    beg = np.arange(V + 1, dtype=np.uint64) * deg
    eb = beg[vb]
    slot = max(sizes) * 4 + 64
    cache = (V + 1) * 8 + (1 + prefetch) * slot * 5 // 8 + 3 * slot
    assert cache < (V + 1) * 8 + 4 * len(csr)
    eng = gw.WalkEngine(algorithm=0, maxhops=5, p=0.5, q=2.0, seed=4, walkpersource=1, compress_blocks=1,
                        prefetch=prefetch, cache_size=cache)
    eng.set_host_graph(beg, csr, vb, eb)
    eng.init_walkers(0, 1, 4)
    st = eng.run()
    ref = oracle.walk(beg, csr, oracle.make_cfg(algo=0, maxhops=5, p=0.5, q=2.0, seed=4, wps=1), 0, V, paths=False)
    assert st["block_loads"] > 0
    assert np.array_equal(eng.hashes(), ref["hashes"])
    eng.close()
