"""Rows of the warp-per-pixel kernel, bit for bit against the oracle in both
modes: delays per level from 1 to more than a warp has lanes for, row lengths
at the edges of its launches, series whose levels end inside a word of four
bins and at its end, rows from nearly full to one event in 40 bins, rows packed
into one part of the series (their buffer falls out of order at the high
levels), counts that reach 255, 256 and more at one level or another, and
values below zero."""
import numpy as np
import pytest

import oracle
import xpcs_gpu as xg
from fixtures import same_bits

pytestmark = pytest.mark.gpu

LENGTHS = (113, 150, 255, 256, 257, 400, 700, 1023, 1024, 1025, 1500, 4000, 4096, 4097)
# name: (frames, dpl, lowest value, one past the highest)
CASES = {
    "dpl_1": (1001, 1, 1, 4),
    "dpl_2": (2050, 2, 1, 4),
    "dpl_4": (4099, 4, 1, 4),
    "dpl_8": (4096, 8, 1, 4),
    "dpl_9": (3001, 9, 1, 4),
    "dpl_16": (2500, 16, 1, 4),
    "dpl_20": (2500, 20, 1, 4),
    "dpl_33": (1200, 33, 1, 3),
    "long": (12345, 8, 1, 3),
    "short": (301, 4, 1, 3),
    "counts_to_255": (1503, 4, 250, 256),
    "counts_past_255": (1502, 8, 100, 300),
    "counts_below_zero": (1500, 4, -3, 5),
}


@pytest.mark.parametrize("mode", [xg.MODE_REFERENCE, xg.MODE_EXACT])
@pytest.mark.parametrize("name", sorted(CASES))
def test_warp_rows_vs_oracle(name, mode):
    F, dpl, lo, hi = CASES[name]
    W, H = 31, 23
    rng = np.random.default_rng(F + dpl)
    P = W * H
    pix, frame = [np.arange(P)], [rng.integers(0, F, P)]  # one event elsewhere
    lengths = [n for n in LENGTHS if n <= F]
    for j, n in enumerate(lengths):
        # spread out, in the first part, in the last part, in two parts
        parts = (np.arange(F), np.arange(min(F, 3 * n)), np.arange(max(0, F - 2 * n), F),
                 np.r_[0:min(F, n // 2 + 9), F - n // 2 - 9:F])
        for k, bins in enumerate(parts):
            bins = np.unique(bins[(bins >= 0) & (bins < F)])
            n1 = min(n, bins.size)
            pix.append(np.full(n1, 4 * j + k + 40))
            frame.append(rng.choice(bins, n1, replace=False))
    key = np.unique(np.concatenate(frame).astype(np.int64) * P + np.concatenate(pix))
    nnz = np.bincount(key // P, minlength=F).astype(np.uint32)
    idx = (key % P).astype(np.int32)
    val = rng.integers(lo, hi, idx.size).astype(np.int16)
    dq = np.ones((H, W), np.int32)
    with xg.Series(W, H, F, dpl, dq, dq) as s:
        s.ingest_sparse(nnz, idx, val)
        s.multitau(mode)
        got = s.g2ipif()
    rows, _ = oracle.sparse_filter(oracle.QMap(dq, dq), nnz, idx, val, F)
    want = oracle.multitau2(rows, F, dpl, mode)
    for g, w, which in zip(got, want, ("G2", "IP", "IF")):
        assert same_bits(g, w), (which, int(np.count_nonzero(g != w)))
