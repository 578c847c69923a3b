"""LZMA2 second stage where its run ends, caps and carries can go wrong: runs
that cross lanes, 128-position blocks and warp ranges, lengths around the cap
of 273, 2- and 3-byte matches, the window's last bytes; every thread count."""
import numpy as np
import pytest

from oracle import oracle as orc

pytestmark = pytest.mark.gpu


def _flipped(n, seed, period, gap):
    rng = np.random.default_rng(seed)
    d = np.resize(rng.integers(0, 256, period, dtype=np.uint8), n).copy()
    at = np.cumsum(rng.integers(1, 2 * gap, n // gap + 1))
    at = at[at < n]
    d[at] ^= rng.integers(1, 256, at.size, dtype=np.uint8)
    return d


DATA = [(1, 5), (1, 274), (2, 130), (4, 400), (5, 17), (127, 60), (128, 277), (129, 1000), (700, 90), (5000, 300)]


@pytest.mark.parametrize("threads", [256, 512, 1024])
@pytest.mark.parametrize("period,gap", DATA)
def test_lzma2_runs_vs_oracle(ctx, period, gap, threads):
    ctx.set_option("lzma_threads", threads)
    try:
        for depth in (0, 32):
            for i, n in enumerate((2, 3, 7, 127, 128, 129, 130, 257, 4096 + 3, 65536, 2 * 65536 + 1027)):
                data = _flipped(n, 7 * i + period, period, gap)
                packed, has = ctx.lzma2_match_find(data, depth)
                o = orc.lzma_packed(data, depth)
                np.testing.assert_array_equal(packed, o)
                np.testing.assert_array_equal(has, orc.has_matches(o, n))
    finally:
        ctx.set_option("lzma_threads", 1024)
