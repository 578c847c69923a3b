"""The compaction of the GPU frames: frames of every small size and alignment
land back to back, raw ones (copied from the window) and compressed ones
(copied from their slot), with one and with several CTAs per window."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("count", [40, 1100])
def test_frames_of_every_alignment_decode(ctx, count):
    from gcz import codecs

    rng = np.random.default_rng(count)
    files = []
    for i in range(count):
        n = int(rng.integers(1, 400)) if count > 1000 else 1 + i * 997
        if i % 3 == 0:
            files.append(rng.integers(0, 256, n, dtype=np.uint8))
        else:
            files.append(np.resize(rng.integers(97, 105, 50 + i % 40, dtype=np.uint8), n))
    res = ctx.zstd_compress_files_gpu(files, 1)
    ends = np.cumsum([len(f) for frames in res for f in frames]) % 16
    assert count < 1000 or set(ends.tolist()) == set(range(16))
    for f, frames in zip(files, res):
        assert b"".join(codecs.zstd_decompress(fr, 65536) for fr in frames) == f.tobytes()
