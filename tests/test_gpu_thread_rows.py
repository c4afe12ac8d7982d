"""Rows of the thread-per-pixel kernel, bit for bit against the oracle in both
modes: delays per level below, at and above what the byte products of the denser
levels take, row capacities from the smallest to the largest, series whose
levels end inside a word of four bins and at its end, the last frame that fits
16 bits, rows that are spread out, packed into one part of the series or into
two (their buffer falls out of order at the high levels), empty and full rows,
counts that reach 255, 256 and more at one level or another in some lanes of a
warp, and values below zero.  The same rows also as a series of few pixels takes
them by itself, a warp a row."""
import numpy as np
import pytest

import oracle
import xpcs_gpu as xg
from fixtures import same_bits

pytestmark = pytest.mark.gpu

# name: (frames, dpl, mean row length, lowest value, one past the highest)
CASES = {
    "dpl_1": (501, 1, 10, 1, 4),
    "dpl_2": (1030, 2, 20, 1, 4),
    "dpl_3": (777, 3, 30, 1, 4),
    "dpl_4": (1000, 4, 10, 1, 4),
    "dpl_5": (999, 5, 40, 1, 4),
    "dpl_8": (2048, 8, 50, 1, 4),
    "dpl_9": (1003, 9, 50, 1, 4),
    "dpl_16": (2500, 16, 30, 1, 4),
    "long": (20000, 8, 60, 1, 3),
    "65536_frames": (65536, 8, 20, 1, 3),
    "short": (61, 4, 15, 1, 3),
    "full": (100, 4, 70, 1, 3),
    "counts_to_255": (402, 4, 9, 60, 256),
    "counts_past_255": (1502, 8, 20, 1, 200),
    "counts_below_zero": (1500, 4, 40, -2, 4),
}


@pytest.mark.parametrize("rows", ["thread", "warp"])
@pytest.mark.parametrize("mode", [xg.MODE_REFERENCE, xg.MODE_EXACT])
@pytest.mark.parametrize("name", sorted(CASES))
def test_thread_rows_vs_oracle(name, mode, rows):
    F, dpl, mean, lo, hi = CASES[name]
    W, H = 53, 31
    rng = np.random.default_rng(F + dpl)
    P = W * H
    pix, frame = [], []
    for p in range(P):
        n = min(int(rng.poisson(mean)), F)
        if p % 97 < 3:
            n = (0, 1, min(F, 2 * mean))[p % 97]
        bins = (np.arange(F), np.arange(min(F, 2 * n)), np.arange(max(0, F - 2 * n), F),
                np.r_[0:min(F, n // 2 + 3), max(0, F - n // 2 - 3):F])[int(rng.integers(4))]
        bins = np.unique(bins)
        n = min(n, bins.size)
        pix.append(np.full(n, p))
        frame.append(rng.choice(bins, n, replace=False))
    key = np.unique(np.concatenate(frame).astype(np.int64) * P + np.concatenate(pix))
    nnz = np.bincount(key // P, minlength=F).astype(np.uint32)
    idx = (key % P).astype(np.int32)
    val = rng.integers(lo, hi, idx.size).astype(np.int16)
    if name == "counts_past_255":  # in a few lanes only
        val = np.where(idx % 41 == 3, val, 1).astype(np.int16)
    dq = np.ones((H, W), np.int32)
    with xg.Series(W, H, F, dpl, dq, dq) as s:
        if rows == "thread":  # else the few pixels of this detector take a warp a row
            s.set_tuning(next(c for c in (32, 48, 64, 80, 112) if c >= 1.5 * mean or c == 112))
        s.ingest_sparse(nnz, idx, val)
        s.multitau(mode)
        got = s.g2ipif()
    events, _ = oracle.sparse_filter(oracle.QMap(dq, dq), nnz, idx, val, F)
    want = oracle.multitau2(events, F, dpl, mode)
    for g, w, which in zip(got, want, ("G2", "IP", "IF")):
        assert same_bits(g, w), (which, int(np.count_nonzero(g != w)))
