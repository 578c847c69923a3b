"""The Zstd lane parse (parse_seg 1024) at the edges of its segments, lists and
mends, against the oracle: ragged sizes, long matches over many segments,
regular data whose parses join late, and data dense in repeat offsets."""
import numpy as np
import pytest

from oracle import oracle as orc

pytestmark = pytest.mark.gpu


def _records(n, seed):
    """Fixed-stride records: repeat offsets decide most matches."""
    rng = np.random.default_rng(seed)
    k = n // 20 + 1
    r = np.zeros(k, dtype=[("id", "<u4"), ("t", "<u4"), ("x", "<f4"), ("f", "u1"), ("s", "S7")])
    r["id"] = np.arange(k)
    r["t"] = 10**9 + np.cumsum(rng.integers(0, 50, k))
    r["x"] = rng.normal(size=k)
    r["f"] = rng.integers(0, 4, k)
    r["s"] = [b"name%02d" % i for i in rng.integers(0, 50, k)]
    return np.frombuffer(r.tobytes(), np.uint8)[:n].copy()


def _csv(n, seed):
    rng = np.random.default_rng(seed)
    lines = b"\n".join(b"%d,user%d,%.3f,%d" % (i, rng.integers(1000), rng.normal(), rng.integers(100))
                       for i in range(n // 20 + 1))
    return np.frombuffer(lines, np.uint8)[:n].copy()


def _periodic(n, seed, period, gap):
    """A period with a changed byte every `gap` bytes or so."""
    rng = np.random.default_rng(seed)
    d = np.resize(rng.integers(0, 256, period, dtype=np.uint8), n).copy()
    at = np.cumsum(rng.integers(1, 2 * gap, n // gap + 1))
    at = at[at < n]
    d[at] = rng.integers(0, 256, at.size, dtype=np.uint8)
    return d


def _walk(n, seed, step):
    return np.cumsum(np.random.default_rng(seed).integers(-step, step + 1, n)).astype(np.uint8)


CASES = [("records", _records, ()), ("csv", _csv, ()), ("zeros", _periodic, (1, 10**7)), ("runs", _periodic, (1, 300)),
         ("p3", _periodic, (3, 40)), ("p7", _periodic, (7, 11)), ("p129", _periodic, (129, 100)),
         ("p300", _periodic, (300, 5000)), ("p1000", _periodic, (1000, 60)), ("walk1", _walk, (1,)), ("walk2", _walk, (2,))]


@pytest.mark.parametrize("depth", [1, 16])
@pytest.mark.parametrize("name,make,args", CASES, ids=[c[0] for c in CASES])
def test_lane_parse_vs_oracle(ctx, name, make, args, depth):
    for i, n in enumerate((1, 3, 4, 5, 127, 128, 129, 131, 132, 133, 259, 4096, 65535, 65536 + 130, 6 * 65536 + 12345)):
        data = make(n, 100 + i, *args)
        seqs, offsets = ctx.zstd_match_find(data, depth)
        o_seqs, o_off = orc.zstd_sequences(data, depth, threads=8)
        np.testing.assert_array_equal(offsets, o_off)
        np.testing.assert_array_equal(seqs, o_seqs)


@pytest.mark.parametrize("max_seqs", [1, 3, 100, 1500])
def test_lane_parse_capped(ctx, max_seqs):
    """A capped parse with repeat-offset matches before and after the cap
    (reference layout: the caller chooses the stride)."""
    import torch as t

    for data in (_csv(2 * 65536 + 77, 5), _periodic(3 * 65536, 6, 7, 11)):
        n = data.size
        B = (n + 65535) // 65536
        d_in = t.from_numpy(data).cuda()
        seqs = t.zeros(B * max_seqs * 3, dtype=t.int32, device="cuda")
        sc, lc = (t.zeros(B, dtype=t.int32, device="cuda") for _ in range(2))
        st = t.cuda.current_stream().cuda_stream
        ctx.zstd_match_find_ref_layout_device(d_in.data_ptr(), seqs.data_ptr(), None, sc.data_ptr(), lc.data_ptr(),
                                              65536, B, n, 16, max_seqs, st)
        ctx.sync(st)
        o = orc.zstd_ref_layout(data, 16, 65536, max_seqs, literals=False)
        o_seqs, o_sc, o_lc = o[0], o[-2], o[-1]
        sc, lc = sc.cpu().numpy(), lc.cpu().numpy()
        np.testing.assert_array_equal(sc, o_sc)
        np.testing.assert_array_equal(lc, o_lc)
        got, want = seqs.cpu().numpy().reshape(B, max_seqs, 3), np.asarray(o_seqs).reshape(B, max_seqs, 3)
        for b in range(B):
            np.testing.assert_array_equal(got[b, :sc[b]], want[b, :sc[b]])
