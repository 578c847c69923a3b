"""The candidate sweep at the edges of its chunks, turns and epochs: seen
through the LZMA2 matches, which show every position's candidate."""
import numpy as np
import pytest

from oracle import oracle as orc

pytestmark = pytest.mark.gpu

CHUNK = 512  # positions of one turn


def _data(kind, n):
    rng = np.random.default_rng(n)
    if kind == "zeros":
        return np.zeros(n, np.uint8)
    if kind == "period":  # equal hashes inside every step
        return np.resize(rng.integers(0, 256, 5, dtype=np.uint8), n)
    if kind == "few":
        return rng.integers(0, 3, n, dtype=np.uint8)
    return rng.integers(0, 256, n, dtype=np.uint8)


@pytest.mark.parametrize("warps,groups", [(7, 0), (6, 0), (5, 0), (4, 0), (7, 1), (4, 1)])
@pytest.mark.parametrize("kind", ["zeros", "period", "few", "random"])
def test_sweep_edges(ctx, kind, warps, groups):
    ctx.set_option("sweep_warps", warps)
    ctx.set_option("sweep_groups", groups)
    try:
        for n in (1, 3, 4, 5, CHUNK - 1, CHUNK, CHUNK + 1, CHUNK + 3, CHUNK + 4, 7 * CHUNK + 2, 65535, 65536,
                  65536 + CHUNK + 1, 500 * 65536 + 77):
            if n > 1 << 20 and groups:
                n = 9 * 65536 + 77
            data = _data(kind, n)
            packed, _ = ctx.lzma2_match_find(data, 32)
            np.testing.assert_array_equal(packed, orc.lzma_packed(data, 32, threads=16))
    finally:
        ctx.set_option("sweep_warps", 7)
        ctx.set_option("sweep_groups", 0)


def test_sweep_epoch_wrap(ctx):
    """More windows per CTA than the table's epochs: 16-byte windows whose
    content repeats every 2^16 windows have to give repeating matches."""
    import torch as t

    sms = t.cuda.get_device_properties(0).multi_processor_count
    period = 1 << 16
    reps = 3 * sms + 1  # 3 CTAs per SM, 65535 epochs each
    block = np.random.default_rng(3).integers(0, 2, period * 16, dtype=np.uint8)
    d_in = t.from_numpy(block).cuda().repeat(reps)
    n, nw = d_in.numel(), period * reps
    m = t.zeros(n * 2, dtype=t.int32, device="cuda")
    c = t.zeros(n, dtype=t.int32, device="cuda")
    st = t.cuda.current_stream().cuda_stream
    ctx.lzma2_match_find_ref_layout_device(d_in.data_ptr(), m.data_ptr(), c.data_ptr(), 16, nw, n, 1, 32, st)
    ctx.sync(st)
    om, oc = orc.lzma_ref_layout(block, 1, 32, window=16)
    assert t.equal(c.view(reps, -1), t.from_numpy(oc.view(np.int32)).cuda().expand(reps, -1))
    assert t.equal(m.view(reps, -1), t.from_numpy(om.reshape(-1).view(np.int32)).cuda().expand(reps, -1))
