"""A borrowed CSR that is written between runs: every run walks what the arrays
hold when it begins, whatever the handle keeps from the run before."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def graph_of(degrees, rng):
    V = len(degrees)
    beg = np.zeros(V + 1, np.uint64)
    beg[1:] = np.cumsum(degrees)
    csr = np.concatenate([np.sort(rng.integers(0, V, d)) for d in degrees]).astype(np.uint32)
    return beg, csr


def expect(eng, st, oracle, beg, csr, algo, term, p, q):
    cfg = oracle.make_cfg(algo=algo, maxhops=30, p=p, q=q, alpha=0.2, term_prob=term, seed=9, wps=4)
    ref = oracle.walk(beg, csr, cfg, 0, 4 * (len(beg) - 1), paths=False)
    assert np.array_equal(eng.hashes(), ref["hashes"])
    assert (st["steps"], st["trials"]) == (ref["stats"]["steps"], ref["stats"]["trials"])


@pytest.mark.parametrize("degrees", ["low", "wide"])
@pytest.mark.parametrize("algo,p,q,offset", [(0, 0.5, 2.0, 0), (0, 2.0, 0.5, 3), (0, 0.25, 4.0, 0), (1, 0.5, 2.0, 0),
                                             (0, 1.0, 1.0, 0)])
def test_writes_between_runs_are_walked(gw, oracle, degrees, algo, p, q, offset):
    import torch
    rng = np.random.default_rng(2)
    V, term = 3000, 0.15 if algo else 0.0
    deg = rng.integers(2, 14, V) if degrees == "low" else np.minimum(rng.zipf(1.7, V) + 1, 900)
    beg, csr = graph_of(deg, rng)
    d_beg = torch.from_numpy(beg.view(np.int64)).cuda()
    d_csr = torch.zeros(len(csr) + 8, dtype=torch.int32, device="cuda")
    eng = gw.WalkEngine(algorithm=algo, maxhops=30, p=p, q=q, alpha=0.2, term_prob=term, seed=9, walkpersource=4)

    def write(beg, csr):
        d_beg.copy_(torch.from_numpy(beg.view(np.int64)))
        d_csr[offset:offset + len(csr)] = torch.from_numpy(csr.view(np.int32)).cuda()
        torch.cuda.synchronize()

    def run():
        eng.init_walkers()
        return eng.run()

    write(beg, csr)
    eng.set_device_graph(V, len(csr), d_beg.data_ptr(), d_csr.data_ptr() + 4 * offset)
    for _ in range(2):
        expect(eng, run(), oracle, beg, csr, algo, term, p, q)
    # other neighbours, the same degrees
    beg2, csr2 = graph_of(deg, rng)
    write(beg2, csr2)
    expect(eng, run(), oracle, beg2, csr2, algo, term, p, q)
    expect(eng, run(), oracle, beg2, csr2, algo, term, p, q)
    # other degrees
    beg3, csr3 = graph_of(rng.permutation(deg), rng)
    write(beg3, csr3)
    expect(eng, run(), oracle, beg3, csr3, algo, term, p, q)
    # one id of one list
    csr4 = csr3.copy()
    v = int(np.argmax(np.diff(beg3.astype(np.int64))))
    csr4[int(beg3[v + 1]) - 1] = V - 1
    write(beg3, csr4)
    expect(eng, run(), oracle, beg3, csr4, algo, term, p, q)
    eng.close()


def test_weights_and_offsets_written_and_given_again(gw, oracle):
    import torch
    rng = np.random.default_rng(4)
    V = 2500
    deg = np.minimum(rng.zipf(1.7, V) + 1, 700)
    beg, csr = graph_of(deg, rng)
    d = [torch.from_numpy(x.copy()).cuda() for x in (beg.view(np.int64), csr.view(np.int32), np.ones(len(csr), np.float32))]
    eng = gw.WalkEngine(algorithm=0, maxhops=30, p=0.5, q=2.0, seed=9, walkpersource=4)
    eng.set_device_graph(V, len(csr), d[0].data_ptr(), d[1].data_ptr())
    for k in range(3):
        beg, csr = graph_of(rng.permutation(deg), rng)
        w = rng.lognormal(0, 1, len(csr)).astype(np.float32)
        for t, x in zip(d, (beg.view(np.int64), csr.view(np.int32), w)):
            t.copy_(torch.from_numpy(x))
        torch.cuda.synchronize()
        eng.set_device_weights(d[2].data_ptr())
        for _ in range(2):
            eng.init_walkers()
            eng.run()
            ref = oracle.walk(beg, csr, oracle.make_cfg(algo=0, maxhops=30, p=0.5, q=2.0, seed=9, wps=4), 0, 4 * V,
                              paths=False, alias=oracle.build_alias(beg, w))
            assert np.array_equal(eng.hashes(), ref["hashes"])
    eng.close()


@pytest.mark.parametrize("count", [300, 12000])
def test_writes_on_the_engine_stream_are_waited_for(gw, oracle, count):
    """The new arrays arrive on the engine's own stream, behind work that takes a while."""
    import torch
    rng = np.random.default_rng(5)
    V = 3000
    beg, csr = graph_of(rng.integers(2, 30, V), rng)
    beg2, csr2 = graph_of(rng.permutation(np.diff(beg.astype(np.int64))), rng)
    d = [torch.from_numpy(x.copy()).cuda() for x in (beg.view(np.int64), csr.view(np.int32))]
    new = [torch.from_numpy(x.copy()).cuda() for x in (beg2.view(np.int64), csr2.view(np.int32))]
    busy = torch.zeros(1 << 28, dtype=torch.float32, device="cuda")
    eng = gw.WalkEngine(algorithm=0, maxhops=30, p=0.5, q=2.0, seed=9, walkpersource=4)
    eng.set_device_graph(V, len(csr), d[0].data_ptr(), d[1].data_ptr())
    stream = torch.cuda.ExternalStream(eng.stream_handle())
    eng.init_walkers(first=0, count=count)
    eng.run()
    torch.cuda.synchronize()
    with torch.cuda.stream(stream):
        for _ in range(8):
            busy.add_(1.0)
        d[0].copy_(new[0])
        d[1].copy_(new[1])
    eng.run()
    cfg = oracle.make_cfg(algo=0, maxhops=30, p=0.5, q=2.0, seed=9, wps=4)
    assert np.array_equal(eng.hashes(), oracle.walk(beg2, csr2, cfg, 0, count, paths=False)["hashes"])
    eng.close()


def test_an_invalid_write_is_refused(gw, oracle):
    import torch
    rng = np.random.default_rng(3)
    beg, csr = graph_of(rng.integers(1, 9, 2000), rng)
    d_beg, d_csr = torch.from_numpy(beg.view(np.int64)).cuda(), torch.from_numpy(csr.view(np.int32)).cuda()
    eng = gw.WalkEngine(algorithm=0, maxhops=30, p=0.5, q=2.0, seed=9, walkpersource=4)
    eng.set_device_graph(2000, len(csr), d_beg.data_ptr(), d_csr.data_ptr())
    eng.init_walkers()
    expect(eng, eng.run(), oracle, beg, csr, 0, 0.0, 0.5, 2.0)
    d_csr[77] = 2000
    torch.cuda.synchronize()
    with pytest.raises(gw.GwError) as e:
        eng.run()
    assert e.value.status == -7
    d_csr.copy_(torch.from_numpy(csr.view(np.int32)))
    torch.cuda.synchronize()
    expect(eng, eng.run(), oracle, beg, csr, 0, 0.0, 0.5, 2.0)
    eng.close()
