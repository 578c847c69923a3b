"""The Huffman plan of the GPU frames on literal counts that are hard for it:
ties, sums that meet other weights, deep trees cut to 11 bits, two bytes, and
FSE-coded weights of every length; frames byte for byte against the restatement."""
import numpy as np
import pytest

import zstd_frames_ref as zr
from oracle import oracle as orc

pytestmark = pytest.mark.gpu

W = 65536


def _counts(kind, n, rng):
    i = np.arange(n, dtype=float)
    if kind == "equal":
        return np.ones(n)
    if kind == "powers":
        return 2.0 ** (i % 12)
    if kind == "steep":
        return 1.6 ** np.minimum(i, 22)
    if kind == "one":
        return np.where(i == 0, 40.0 * n, 1.0)
    if kind == "zipf":
        return 1.0 / (1.0 + i)
    return rng.integers(1, 200, n).astype(float)


@pytest.mark.parametrize("kind", ["equal", "powers", "steep", "one", "zipf", "mixed"])
def test_plans_equal_reference(ctx, kind):
    rng = np.random.default_rng(21)
    wins = []
    for n in (2, 3, 5, 31, 33, 100, 128, 129, 130, 131, 200, 255, 256):
        c = _counts(kind, n, rng)
        size = int(rng.choice([W, W, 3000, 20011])) if wins else W
        c = np.maximum(1, np.floor(c / c.sum() * size)).astype(int)
        vals = rng.permutation(256)[:n] if n < 256 else np.arange(256)
        d = rng.permutation(np.repeat(vals, c))[:size].astype(np.uint8)
        wins.append(d)
    res = ctx.zstd_compress_files_gpu(wins, 1)
    for d, frames in zip(wins, res):
        seqs, _ = orc.zstd_sequences(d, 16)
        assert len(frames) == 1 and bytes(frames[0]) == zr.encode_frame(d.tobytes(), [(x[0], x[1], x[2]) for x in seqs])
