"""Offsets of a CSR built on the device where vertices without edges lie in a
row: gaps around the length a thread fills by itself and the length of a piece,
before the first source, between sources and past the last, and more offsets
than the scratch of a few edges holds."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nverts,sources", [
    (1, []),
    (130, [0, 64, 129]),
    (5000, np.cumsum([63, 64, 65, 66, 1, 2, 64, 1023, 1024, 1025, 1088])),
    (1 << 20, [0]),
    (1 << 20, [(1 << 20) - 1]),
    (3_000_000, np.cumsum([1_000_003, 1, 64, 999_999, 65])),
    (200_000, np.arange(0, 200_000, 65)),
    (200_000, np.arange(70, 200_000, 97)),
])
@pytest.mark.parametrize("sort", [True, False])
def test_offsets_over_gaps(gw, nverts, sources, sort):
    src = np.repeat(np.asarray(sources, np.uint32), 3)
    dst = np.tile(np.asarray([2, 7, 9], np.uint32), len(sources)) % max(nverts, 1)
    dst = np.where(dst == src, (dst + 1) % max(nverts, 1), dst).astype(np.uint32)
    order = np.random.default_rng(1).permutation(len(src))
    g = gw.DeviceGraph.from_edges(src[order], dst[order], nverts=nverts, sort=sort)
    beg, csr = g.to_host()
    want = np.zeros(nverts + 1, np.uint64)
    want[1:] = np.cumsum(np.bincount(src, minlength=nverts))
    assert np.array_equal(beg, want)
    for v in np.asarray(sources, np.int64)[:50]:
        assert sorted(csr[int(beg[v]):int(beg[v + 1])]) == sorted(dst[src == v])
