"""Side statistics over the integer pass and the ordered one, bit for bit
against the oracle: frame counts around the chunk of a warp, windows that do
not divide the series, one-frame windows, more frames than the shared-memory
counters hold, bins and frames whose sums pass 2^24, a total past 2^32 and
negative counts (all three: the ordered sums)."""
import numpy as np
import pytest

import oracle
import xpcs_gpu as xg
from fixtures import same_bits_nan

pytestmark = pytest.mark.gpu

# name: (W, H, frames, static window, mean, lowest count, highest count)
CASES = {
    "one_frame": (9, 7, 1, 1, 0.5, 1, 3),
    "window_1": (8, 9, 33, 1, 0.6, 1, 4),
    "window_7_of_31": (33, 5, 31, 7, 0.4, 1, 2),
    "window_past_the_end": (16, 16, 20, 64, 0.3, 0, 5),
    "30000_frames": (5, 5, 30000, 3000, 0.05, 1, 3),
    "many_windows": (6, 6, 9000, 2, 0.1, 1, 3),
    "sums_past_2_24": (16, 12, 60, 9, 0.9, 20000, 32767),
    "total_past_2_32": (40, 40, 120, 120, 0.95, 30000, 32767),
    "negative": (16, 12, 60, 9, 0.3, -5, 9),
}


@pytest.mark.parametrize("name", sorted(CASES))
def test_side_statistics_vs_oracle(name):
    W, H, F, win, mean, lo, hi = CASES[name]
    rng = np.random.default_rng(len(name))
    P = W * H
    sq = (np.arange(P, dtype=np.int32) * 4 // P) + 1
    dq = (sq + 1) // 2
    dq[rng.random(P) < 0.1] = 0
    hit = rng.random((F, P)) < mean
    nnz, idx = hit.sum(1).astype(np.uint32), np.nonzero(hit)[1].astype(np.int32)
    val = rng.integers(lo, hi + 1, idx.size).astype(np.int16)
    with xg.Series(W, H, F, 4, dq.reshape(H, W), sq.reshape(H, W), static_window=win) as s:
        s.ingest_sparse(nnz, idx, val)
        s.multitau()
        ps, fs, tot, part = s.side_stats(win)
    qm = oracle.QMap(dq.reshape(H, W), sq.reshape(H, W))
    _, side = oracle.sparse_filter(qm, nnz, idx, val, F, static_window=win)
    assert same_bits_nan(ps.ravel(), side["pixels_sum"].ravel())
    assert same_bits_nan(fs.ravel(), side["frames_sum"].ravel())
    assert same_bits_nan(tot.ravel(), side["partitions_mean"].ravel())
    assert same_bits_nan(part.ravel(), side["partial_mean"].ravel()[:part.size])
