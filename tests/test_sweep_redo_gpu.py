"""The candidate sweep's check of its own order: an order that it does not expect
is found and the windows are swept again, after the table has been used and
candidates have been written.  And its former grouping option costs nothing."""
import numpy as np
import pytest

import gcz
from oracle import oracle as orc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["bench", "period", "random", "mixed"])
def test_redo_vs_oracle(ctx, kind):
    import torch as t

    sms = t.cuda.get_device_properties(0).multi_processor_count
    for n in (4, 33, 515, 4096, 65536, 9 * 65536 + 77, (7 * sms + 3) * 65536 + 5):  # up to three windows per CTA
        rng = np.random.default_rng(n)
        data = {"bench": lambda: orc.gen_synthetic(3, n),
                "period": lambda: np.resize(rng.integers(0, 256, 5, dtype=np.uint8), n),
                "random": lambda: rng.integers(0, 256, n, dtype=np.uint8),
                "mixed": lambda: np.where(np.arange(n) // 65536 % 3 == 1, 7, rng.integers(0, 256, n)).astype(np.uint8),
                }[kind]()
        d = t.from_numpy(data).cuda()
        packed = t.zeros(n, dtype=t.int32, device="cuda")
        has = t.zeros((n + 65535) // 65536, dtype=t.uint8, device="cuda")
        st = t.cuda.current_stream().cuda_stream or 1
        assert gcz.L.gcz_selftest_sweep_redo(ctx.handle, d.data_ptr(), n, 32, packed.data_ptr(), has.data_ptr(), st) == 0
        ctx.sync(t.cuda.current_stream().cuda_stream)
        np.testing.assert_array_equal(packed.cpu().numpy().view(np.uint32), orc.lzma_packed(data, 32, threads=16))


def test_grouping_option_costs_nothing(ctx):
    import torch as t

    n = 64 << 20
    d = t.from_numpy(orc.gen_synthetic(4, n)).cuda()
    packed = t.zeros(n, dtype=t.int32, device="cuda")
    has = t.zeros(n // 65536, dtype=t.uint8, device="cuda")
    st = t.cuda.current_stream().cuda_stream

    def best():
        ms = []
        for _ in range(6):
            a, b = (t.cuda.Event(enable_timing=True) for _ in range(2))
            a.record()
            ctx.lzma2_match_find_device(d.data_ptr(), n, 32, packed.data_ptr(), has.data_ptr(), st)
            b.record()
            b.synchronize()
            ms.append(a.elapsed_time(b))
        return min(ms[1:])

    try:
        base = best()
        for groups in (1, 2, 3):
            ctx.set_option("sweep_groups", groups)
            assert ctx.query("sweep_groups") == groups
            assert best() <= 1.25 * base
    finally:
        ctx.set_option("sweep_groups", 0)
