"""A handle that is given another graph walks that one: nothing sized for the
graph before is used, whichever is the larger."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scales", [(9, 15), (15, 9, 14)])
@pytest.mark.parametrize("device", [False, True])
def test_weighted_walks_after_another_graph(gw, oracle, scales, device):
    import torch
    eng = gw.WalkEngine(algorithm=0, maxhops=15, p=2.0, q=0.5, seed=6, record_paths=0)
    for scale in scales:
        beg, csr = oracle.rmat_graph(scale, seed=scale)
        V = len(beg) - 1
        w = np.random.default_rng(scale).lognormal(0.0, 1.0, len(csr)).astype(np.float32)
        if device:
            d = [torch.from_numpy(beg.view(np.int64)).cuda(), torch.from_numpy(csr.view(np.int32)).cuda(),
                 torch.from_numpy(w).cuda()]
            eng.set_device_graph(V, len(csr), d[0].data_ptr(), d[1].data_ptr())
            eng.set_device_weights(d[2].data_ptr())
        else:
            eng.set_host_graph(beg, csr)
            eng.set_host_weights(w)
        eng.init_walkers(0, 1, 6)
        eng.run()
        cfg = oracle.make_cfg(algo=0, maxhops=15, p=2.0, q=0.5, seed=6)
        ref = oracle.walk(beg, csr, cfg, 0, V, paths=False, alias=oracle.build_alias(beg, w))
        assert np.array_equal(eng.hashes(), ref["hashes"])
    eng.close()
