"""Frontier compaction with tiles of 512 and 1024 bitmap words (several words per
thread), which ranges above 8.4 M and 16.8 M vertices get: dense
frontiers of many passes a tile, sparse ones, vertices without edges between,
hubs, ranges that start and end inside a word; the list, the prefix and the
tile map against a numpy model."""
import numpy as np
import pytest

import onegraph_gb300 as og

from test_gpu_kernels import compact_model, run_compact

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.mark.parametrize("V,vb", [
    (8_388_608, 0),        # 1024 tiles of 256 words: the last size before
    (8_388_609, 0),        # 512 words
    (9_000_011, 77),
    (16_777_216, 0),
    (17_000_033, 31),      # 1024 words
    (35_000_000, 32 * 1024 * 7 + 5),
])
@pytest.mark.parametrize("kind", ["dense", "half", "sparse", "clustered"])
def test_wide_tiles(V, vb, kind):
    rng = np.random.default_rng(V)
    deg = rng.integers(0, 4, V)          # a quarter has no edges
    deg[V // 2], deg[V - 1], deg[vb] = 400_000, 5000, 2048
    off = np.concatenate([[0], np.cumsum(deg)]).astype(np.uint64)
    words = (V + 31) // 32
    if kind == "dense":
        bits = np.full(words, 0xFFFFFFFF, np.uint32)
    elif kind == "half":
        bits = rng.integers(0, 1 << 32, words, dtype=np.uint64).astype(np.uint32)
    else:
        bits = np.zeros(words, np.uint32)
        if kind == "sparse":
            ids = rng.integers(0, V, 5000)
            np.bitwise_or.at(bits, ids // 32, np.uint32(1) << (ids % 32).astype(np.uint32))
        else:  # full words in some tiles, nothing in the others
            for s in range(0, words, 2500):
                bits[s:s + 70] = 0xFFFFFFFF
    lst, pref, tiles = compact_model(bits, vb, V, off)
    bits_d = torch.from_numpy(bits.view(np.int32)).cuda()
    off_d = torch.from_numpy(off.view(np.int64)).cuda()
    rc, n, total, (glist, gpref, gtile) = run_compact(bits_d, vb, V, off_d, V, int(off[-1]) // 2048 + 2)
    assert rc == 0, og.lib().og_last_error()
    assert n == lst.size and total == int(pref[-1])
    np.testing.assert_array_equal(glist[:n], lst)
    np.testing.assert_array_equal(gpref[:n + 1], pref)
    np.testing.assert_array_equal(gtile[:tiles.size], tiles)
