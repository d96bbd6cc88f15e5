"""Frontier compaction where its tiles and passes can go wrong: word and tile
remainders, a pass exactly full (2048 listed bits), one more, several passes
with unlisted (zero-degree) vertices between, hubs spanning many edge tiles,
and each tile width."""
import numpy as np
import pytest

import onegraph_gb300 as og

from test_gpu_kernels import compact_model, run_compact

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.mark.parametrize("V,vb,density,zero,hub", [
    (1, 0, 1.0, 0.0, 0),
    (33, 1, 1.0, 0.0, 0),
    (2048, 0, 1.0, 0.0, 0),
    (2049, 0, 1.0, 0.0, 50_000),
    (4096, 0, 1.0, 0.5, 0),
    (4097, 31, 1.0, 0.9, 300_000),
    (70_001, 5, 0.7, 0.3, 100_000),      # 128-word tiles, two passes each
    (70_001, 5, 0.001, 0.0, 0),          # nearly empty tiles
    (5_000_011, 77, 0.9, 0.2, 1_000_000),  # 256-word tiles, four passes
    (5_000_011, 0, 1.0, 1.0, 0),         # nothing listed
])
def test_compact_tiles_and_passes(V, vb, density, zero, hub):
    rng = np.random.default_rng(V)
    deg = rng.integers(1, 12, V).astype(np.uint64)
    deg[rng.random(V) < zero] = 0
    if hub:
        deg[V // 2] = hub
        deg[V - 1] = hub // 3
    off = np.concatenate([[0], np.cumsum(deg)]).astype(np.uint64)
    words = np.packbits(rng.random(((V + 31) // 32) * 32) < density, bitorder="little").view(np.uint32).copy()
    bits_d = torch.from_numpy(words.view(np.int32)).cuda()
    off_d = torch.from_numpy(off.view(np.int64)).cuda()
    lst, pref, tiles = compact_model(words, vb, V, off)
    rc, n, total, (glist, gpref, gtile) = run_compact(bits_d, vb, V, off_d, V, int(off[-1]) // 2048 + 2)
    assert rc == 0, og.lib().og_last_error()
    assert n == lst.size and total == int(pref[-1])
    np.testing.assert_array_equal(glist[:n], lst)
    np.testing.assert_array_equal(gpref[:n + 1], pref)
    np.testing.assert_array_equal(gtile[:tiles.size], tiles)
