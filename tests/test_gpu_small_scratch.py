"""Edge lists and host graphs around the size from which their buffers share an
allocation (1.5 MB): the same CSR, the same walks."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 1000, 98_304, 98_305, 196_576, 196_577, 196_608, 196_609, 400_000])
@pytest.mark.parametrize("symmetric,dedup", [(False, False), (True, True)])
@pytest.mark.parametrize("device", [False, True])
def test_edge_lists_around_one_piece(gw, n, symmetric, dedup, device):
    import torch
    rng = np.random.default_rng(n)
    V = 5003
    src, dst = rng.integers(0, V, n).astype(np.uint32), rng.integers(0, V, n).astype(np.uint32)
    args = [torch.from_numpy(x.view(np.int32)).cuda() for x in (src, dst)] if device else [src, dst]
    g = gw.DeviceGraph.from_edges(*args, nverts=V, symmetric=symmetric, sort=True, dedup=dedup)
    beg, csr = g.to_host()
    keep = src != dst
    k = src[keep].astype(np.uint64) * V + dst[keep]
    if symmetric:
        k = np.concatenate([k, dst[keep].astype(np.uint64) * V + src[keep]])
    k = np.unique(k) if dedup else np.sort(k)
    assert np.array_equal(csr, (k % V).astype(np.uint32))
    assert np.array_equal(np.diff(beg.astype(np.int64)), np.bincount((k // V).astype(np.int64), minlength=V))
    g.free()


@pytest.mark.parametrize("sizes", [(1000, 5000), (196_500, 300_000), (196_700, 300_000), (3000, 393_215), (3000, 393_216)])
def test_host_graphs_around_one_piece(gw, oracle, sizes):
    rng = np.random.default_rng(3)
    eng = gw.WalkEngine(algorithm=0, maxhops=12, p=0.5, q=2.0, seed=2)
    for V, E in (sizes, (500, 2000), sizes):
        deg = np.bincount(rng.integers(0, V, E), minlength=V)
        beg = np.zeros(V + 1, np.uint64)
        beg[1:] = np.cumsum(deg)
        owner = np.repeat(np.arange(V, dtype=np.uint64), deg)
        csr = (np.sort(owner * V + rng.integers(0, V, E).astype(np.uint64)) % V).astype(np.uint32)
        eng.set_host_graph(beg, csr)
        eng.init_walkers()
        eng.run()
        ref = oracle.walk(beg, csr, oracle.make_cfg(algo=0, maxhops=12, p=0.5, q=2.0, seed=2), 0, V, paths=False)
        assert np.array_equal(eng.hashes(), ref["hashes"])
    eng.close()
