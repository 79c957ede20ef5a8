"""How walkers are dealt to warps: populations around what one warp, one CTA an
SM and all lanes hold, sure steps and others, on the device's own grid and on
one that is asked for, walk every walker once."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIZES = [1, 7, 8, 9, 1183, 1184, 1185, 2368, 4736, 4737, 37888, 37889, 75777, 189440, 189441]


@pytest.mark.parametrize("algo,p,q", [(0, 0.5, 2.0), (0, 1.0, 1.0), (0, 0.25, 4.0), (1, 0.5, 2.0)])
@pytest.mark.parametrize("grid", [0, 3, 1000])
def test_every_walker_once(gw, oracle, algo, p, q, grid):
    beg, csr = oracle.rmat_graph(13, seed=8)
    term = 0.15 if algo else 0.0
    sizes = SIZES if grid == 0 else SIZES[::4]
    eng = gw.WalkEngine(algorithm=algo, maxhops=6, p=p, q=q, alpha=0.2, term_prob=term, seed=12, init_mode=2,
                        numwalks=max(sizes), blockpergrid=grid)
    eng.set_host_graph(beg, csr)
    cfg = oracle.make_cfg(algo=algo, maxhops=6, p=p, q=q, alpha=0.2, term_prob=term, seed=12, init_mode=2,
                          numwalks=max(sizes))
    ref = oracle.walk(beg, csr, cfg, 0, max(sizes), paths=False)
    for n in sizes:
        eng.init_walkers(first=0, count=n)
        st = eng.run()
        assert st["walkers"] == n
        assert np.array_equal(eng.hashes(), ref["hashes"][:n])
        assert eng.checksum()[0] == int(ref["hashes"][:n].sum(dtype=np.uint64))
    eng.close()
