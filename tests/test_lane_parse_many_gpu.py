"""The Zstd lane parse has three forms: for at most one window per SM, at most
two, and more.  Each against the oracle, on the data that takes its rarer paths."""
import numpy as np
import pytest

from oracle import oracle as orc
from test_lane_parse_gpu import CASES

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("copies", [1, 6, 12])
def test_each_form_vs_oracle(ctx, copies):
    files = [make(n, 7 + n, *args) for _, make, args in CASES for n in (133, 4096, 65535)]
    assert (len(files) * copies <= 148) == (copies == 1)  # 148 SMs, one window per file
    for depth in (1, 16):
        want = [orc.zstd_sequences(f, depth, threads=1)[0] for f in files]
        seqs, offsets = ctx.zstd_match_find_files(files * copies, depth)
        for i, w in enumerate(want * copies):
            np.testing.assert_array_equal(seqs[int(offsets[i]):int(offsets[i + 1])], w)
