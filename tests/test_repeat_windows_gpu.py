"""Windows whose matches lie mostly at repeat offsets, or whose parses from
different places come together late: what the lane parse cannot mend is parsed
again by lanes with repeat offsets, or by the segment parse.  Against the oracle
in each form of the parse, and timed against the segment parse alone."""
import numpy as np
import pytest

from oracle import oracle as orc

pytestmark = pytest.mark.gpu


def _counters(n, rng):
    """Consecutive 32-bit numbers: every match is three bytes at distance 4."""
    return (np.arange(n // 4 + 1) + 123456789).astype("<u4").view(np.uint8)[:n]


def _sorted_ids(n, rng):
    return np.sort(rng.integers(0, 64 * (n // 4 + 1), n // 4 + 1)).astype("<u4").view(np.uint8)[:n]


def _fields(n, rng, stride):
    """Records of constant bytes but for a 16-bit counter and one random byte."""
    k = np.arange(n // stride + 1)
    r = np.tile(rng.integers(0, 256, stride, dtype=np.uint8), (k.size, 1))
    r[:, 0], r[:, 1], r[:, stride // 2] = k & 255, k >> 8 & 255, rng.integers(0, 256, k.size)
    return r.reshape(-1)[:n]


def _pixels(n, rng):
    return np.cumsum(rng.integers(-1, 2, (n // 3 + 1, 3)), 0).astype(np.uint8).reshape(-1)[:n]


def _wave(n, rng):
    """16-bit samples: few and far between, runs with many repeat-offset matches."""
    k = np.arange(n // 2 + 1)
    return (10000 * np.sin(k / 50) + rng.integers(-20, 20, k.size)).astype("<i2").view(np.uint8)[:n]


def _bases(n, rng):
    """Four symbols: continuations of up to about 60 matches."""
    return np.frombuffer(b"ACGT", np.uint8)[rng.integers(0, 4, n)]


def _floats(n, rng):
    return np.cumsum(rng.normal(size=n // 4 + 1)).astype("<f4").view(np.uint8)[:n]


KINDS = {"counters": (_counters,), "sorted_ids": (_sorted_ids,), "fields8": (_fields, 8), "fields64": (_fields, 64),
         "pixels": (_pixels,), "wave": (_wave,), "bases": (_bases,), "floats": (_floats,)}


def _make(kind, n, seed):
    make, *args = KINDS[kind]
    return np.ascontiguousarray(make(n, np.random.default_rng(seed), *args))


@pytest.mark.parametrize("depth", [1, 16])
@pytest.mark.parametrize("kind", KINDS)
def test_vs_oracle(ctx, kind, depth):
    # one window and less, a few, one per SM (up to 148), two per SM, more (each form of the parse)
    for i, n in enumerate((131, 4096, 65535, 3 * 65536 + 777, 200 * 65536 + 5, 420 * 65536)):
        data = _make(kind, n, 10 + i)
        seqs, offsets = ctx.zstd_match_find(data, depth)
        o_seqs, o_off = orc.zstd_sequences(data, depth, threads=8)
        np.testing.assert_array_equal(offsets, o_off)
        np.testing.assert_array_equal(seqs, o_seqs)


def test_among_other_windows(ctx):
    """Windows given up between windows that are not, several per CTA."""
    n = 700 * 65536
    data = orc.gen_synthetic(5, n)
    for i, kind in enumerate(KINDS):
        for w in range(3 * i + 1, 700, 31):
            data[w * 65536:(w + 1) * 65536] = _make(kind, 65536, i)
    seqs, offsets = ctx.zstd_match_find(data, 16)
    o_seqs, o_off = orc.zstd_sequences(data, 16, threads=8)
    np.testing.assert_array_equal(offsets, o_off)
    np.testing.assert_array_equal(seqs, o_seqs)


@pytest.mark.parametrize("kind", ["counters", "pixels", "wave"])
def test_small_windows_after_given_up_ones(ctx, kind):
    """A CTA that has given up a window gives up the next ones at once: windows of
    a few bytes, of ordinary data and of other kinds among them."""
    import torch as t

    ctas = 3 * t.cuda.get_device_properties(0).multi_processor_count
    rng = np.random.default_rng(9)
    rows = [[_make(kind, 65536 if i % 5 else 4096, i) for i in range(ctas)],
            [rng.integers(0, 3, i % 7, dtype=np.uint8) for i in range(ctas)],
            [orc.gen_synthetic(i, 3000 + i) for i in range(ctas)],
            [_make("bases", 300 + 7 * i, i) for i in range(ctas)],
            [np.zeros(i % 40 + 1, np.uint8) for i in range(ctas)]]
    files = [f for row in rows for f in row]
    seqs, offsets = ctx.zstd_match_find_files(files, 16)
    w = 0
    for f in files:
        if f.size == 0:
            continue
        want = orc.zstd_sequences(f, 16, threads=1)[0]
        np.testing.assert_array_equal(seqs[int(offsets[w]):int(offsets[w + 1])], want)
        w += 1
    assert w + 1 == offsets.size


@pytest.mark.parametrize("kind,windows", [("counters", 16), ("sorted_ids", 16), ("bases", 16), ("fields64", 256),
                                          ("counters", 2048), ("fields8", 2048)])
def test_not_slower_than_segment_parse(ctx, kind, windows):
    """The default schedule is at most a quarter slower than the segment parse
    on windows that it may hand to it (on the same GPU, best of several)."""
    import torch as t

    n = windows * 65536
    d = t.from_numpy(np.resize(_make(kind, min(n, 16 << 20), 3), n)).cuda()
    cap = n // 3
    seqs = t.zeros(cap, 4, dtype=t.int32, device="cuda")
    offs = t.zeros(windows + 1, dtype=t.int64, device="cuda")
    st = t.cuda.current_stream().cuda_stream

    def best():
        ms = []
        for _ in range(6):
            a, b = (t.cuda.Event(enable_timing=True) for _ in range(2))
            a.record()
            for _ in range(3):
                ctx.zstd_match_find_device(d.data_ptr(), n, 16, seqs.data_ptr(), cap, offs.data_ptr(), st)
            b.record()
            b.synchronize()
            ms.append(a.elapsed_time(b))
        return min(ms[1:])

    was = ctx.query("parse_seg")
    try:
        segments = []
        for seg in (2048, 4096, 8192):
            ctx.set_option("parse_seg", seg)
            segments.append(best())
        ctx.set_option("parse_seg", 1024)
        assert best() <= 1.25 * min(segments)
    finally:
        ctx.set_option("parse_seg", was)


def test_sequence_section_of_two_distances(ctx):
    """Encoding a window whose sequences use two distances throughout (the third
    of the repeat history stays from its start) is no slower than one with
    three (same lengths, on the same GPU)."""
    import torch as t

    ns, n = 16000, 65536
    rng = np.random.default_rng(1)
    src = t.from_numpy(rng.integers(0, 256, n, dtype=np.uint8)).cuda()
    offs = t.tensor([0, ns], dtype=t.int64, device="cuda")
    out = t.zeros(2 * n, dtype=t.uint8, device="cuda")
    fo = t.zeros(2, dtype=t.int64, device="cuda")
    st = t.cuda.current_stream().cuda_stream

    def best(off):
        s = np.zeros((ns, 4), np.uint32)  # offset, literals, match length
        s[:, 0], s[:, 1], s[:, 2] = np.minimum(off, 1 + 4 * np.arange(ns)), 1, 3
        d = t.from_numpy(s.view(np.int32)).cuda()
        ms = []
        for _ in range(8):
            a, b = (t.cuda.Event(enable_timing=True) for _ in range(2))
            a.record()
            ctx.zstd_encode_frames_device(src.data_ptr(), n, d.data_ptr(), offs.data_ptr(), out.data_ptr(), 2 * n,
                                          fo.data_ptr(), st)
            b.record()
            b.synchronize()
            ms.append(a.elapsed_time(b))
        ctx.sync(st)
        return min(ms[1:])

    assert best(rng.choice([4, 12], ns)) <= 1.25 * best(rng.choice([4, 12, 20], ns))
