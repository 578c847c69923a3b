"""The sequence section of the GPU Zstd entropy stage at the edges of its
per-thread runs, chunks and tables: made-up sequences (the stage does not look
at what they copy), frames byte for byte against the restatement."""
import numpy as np
import pytest

import zstd_frames_ref as zr

pytestmark = pytest.mark.gpu

W = 65536


def _sequences(kind, ns, rng):
    budget = (W - 64) // ns  # bytes per sequence on average
    if kind == "one":  # every field a single code: RLE_Mode
        ll, ml = np.full(ns, 2), np.full(ns, 5)
        off = np.full(ns, 6)
    elif kind == "skewed":  # one code nearly always: long stretches in which two chains keep apart
        rare = rng.random(ns) < 0.01
        ll, ml = np.where(rare, 1 + rng.integers(0, 3, ns), 1), np.where(rare, 4, 3)
        off = np.where(rare, rng.integers(1, 4, ns), 4)
    elif kind == "repeats":
        ll, ml = rng.integers(0, 2, ns), rng.integers(3, 6, ns)
        off = rng.choice([1, 2, 3, 4, 5, 7], ns)
    else:
        ll = rng.integers(0, max(budget // 2, 1), ns)
        ml = rng.integers(3, max(budget // 2, 4), ns)
        off = 1 + rng.integers(0, 60000, ns)
    out, pos = [], 0
    for a, m, o in zip(ll.tolist(), ml.tolist(), off.tolist()):
        a = max(a, 1) if pos == 0 else a
        if pos + a + m > W:
            break
        out.append((max(1, min(o, pos + a)), a, m))
        pos += a + m
    return out


@pytest.mark.parametrize("kind", ["one", "skewed", "repeats", "mixed"])
def test_sequence_sections_equal_reference(ctx, kind):
    import torch as t

    counts = (1, 2, 3, 31, 32, 33, 127, 128, 129, 255, 1023, 1024, 1025, 1055, 1057, 2048, 2049, 4097)
    rng = np.random.default_rng(11)
    data = rng.choice(np.arange(40, 56, dtype=np.uint8), len(counts) * W, p=np.arange(1, 17) / 136)
    seqs = [_sequences(kind, ns, rng) for ns in counts]
    flat = np.array([(o, a, m, 0) for s in seqs for o, a, m in s], np.uint32)
    offs = np.cumsum([0] + [len(s) for s in seqs]).astype(np.int64)
    d_src, d_seqs, d_off = t.from_numpy(data).cuda(), t.from_numpy(flat.view(np.int32)).cuda(), t.from_numpy(offs).cuda()
    cap = len(counts) * (W + 64)
    d_out = t.zeros(cap, dtype=t.uint8, device="cuda")
    d_fo = t.zeros(len(counts) + 1, dtype=t.int64, device="cuda")
    st = t.cuda.current_stream().cuda_stream
    ctx.zstd_encode_frames_device(d_src.data_ptr(), data.size, d_seqs.data_ptr(), d_off.data_ptr(), d_out.data_ptr(),
                                  cap, d_fo.data_ptr(), st)
    ctx.sync(st)
    out, fo = d_out.cpu().numpy(), d_fo.cpu().numpy()
    for b, s in enumerate(seqs):
        want = zr.encode_frame(data[b * W:(b + 1) * W].tobytes(), s)
        assert out[fo[b]:fo[b + 1]].tobytes() == want, (kind, counts[b])
