"""Small host calls (offsets, records and status written to pinned memory by
the kernels) on both sides of their size limit and of the fused offset scan's."""
import numpy as np
import pytest

from oracle import oracle as orc

pytestmark = pytest.mark.gpu

LIMIT = 256 << 10
W = 65536


@pytest.mark.parametrize("n", [1, 2, 5, 4096, W - 1, W, W + 1, LIMIT - 1, LIMIT, LIMIT + 1, 1024 * W, 1024 * W + 1])
def test_small_host_calls(ctx, n):
    import gcz

    data = gcz.gen_synthetic(n % 1000 + 1, n, 8 << 20)
    o_seqs, o_off = orc.zstd_sequences(data, 16, threads=16)
    seqs, offsets = ctx.zstd_match_find(data, 16)
    np.testing.assert_array_equal(offsets, o_off)
    np.testing.assert_array_equal(seqs, o_seqs)
    recs, offsets = ctx.zstd_match_find_packed(data, 16)
    np.testing.assert_array_equal(offsets, o_off)
    np.testing.assert_array_equal(gcz.expand_packed(recs), o_seqs)


def test_small_host_call_capacity(ctx):
    import gcz

    data = gcz.gen_synthetic(9, 100_000, 8 << 20)
    want, _ = ctx.zstd_match_find(data, 16)
    seqs, offsets = np.full((want.shape[0], 4), 7, np.uint32), np.zeros(3, np.uint64)
    args = (ctx.handle, data.ctypes.data, data.size, 16, seqs.ctypes.data)
    assert gcz.L.gcz_zstd_match_find(*args, want.shape[0] - 1, offsets.ctypes.data) == -4  # GCZ_ECAPACITY
    assert gcz.L.gcz_zstd_match_find(*args, want.shape[0], offsets.ctypes.data) == 0
    np.testing.assert_array_equal(seqs, want)
