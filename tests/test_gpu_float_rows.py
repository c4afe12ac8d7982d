"""Float rows (flatfield, averaging) up to the capacity of the thread-per-pixel
float kernel and past it, bit for bit against the oracle in both modes: delays
per level below, at and above what it takes, rows without events, rows that
fill every frame, rows packed into the first half of the series (their buffer
falls out of order at the high levels), many frames, a detector that ends
inside a window of the kernel's length sort, and one too small for it."""
import numpy as np
import pytest

import oracle
import xpcs_gpu as xg
from fixtures import same_bits

pytestmark = pytest.mark.gpu

# name: (W, H, frames, dpl, average, mean row length, special row lengths)
CASES = {
    "short": (310, 300, 120, 4, 1, 12, (0, 1, 2, 15, 16, 17, 31, 32, 33, *range(74, 90), 120)),
    "mean_40": (310, 300, 400, 8, 1, 40, (63, 64, 65, *range(108, 130), 255, 256, 257, 400)),
    "full": (330, 290, 64, 8, 1, 62, (64, 63, 0, 1)),
    "dpl_9": (310, 300, 100, 9, 1, 20, (64, 65, 100)),
    "dpl_2": (310, 300, 60, 2, 1, 15, (59, 60, 4, 5)),
    "dpl_1": (310, 300, 60, 1, 1, 15, (0, 59, 60)),
    "average_2": (310, 300, 100, 8, 2, 20, (64, 65, 100)),
    "70000_frames": (310, 300, 70000, 8, 1, 5, (64, 65, 71, 72, 300)),
    "small": (19, 13, 500, 8, 1, 80, (1, 63, 64, 65, 223, 224, 225, 500)),
}


@pytest.mark.parametrize("mode", [xg.MODE_REFERENCE, xg.MODE_EXACT])
@pytest.mark.parametrize("name", sorted(CASES))
def test_float_rows_vs_oracle(name, mode):
    W, H, F, dpl, average, mean, special = CASES[name]
    rng = np.random.default_rng(F + dpl)
    P, R = W * H, F * average
    n = rng.poisson(mean, P)
    pix = np.repeat(np.arange(P), n)
    frame = rng.integers(0, R, pix.size)
    early = pix % 11 == 5  # rows in the first half of the series, nearly full
    frame[early] = rng.integers(0, min(R // 2, 2 * mean), np.count_nonzero(early))
    keep = ~np.isin(pix, 7 * np.arange(len(special)))
    pix, frame = [pix[keep]], [frame[keep]]
    for k, length in enumerate(special):
        pix.append(np.full(length, 7 * k))
        frame.append(rng.choice(F, length, replace=False) * average)
    key = np.unique(np.concatenate(frame).astype(np.int64) * P + np.concatenate(pix))
    nnz = np.bincount(key // P, minlength=R).astype(np.uint32)
    idx = (key % P).astype(np.int32)
    val = rng.integers(1, 6, idx.size).astype(np.int16)
    flat = rng.uniform(0.8, 1.2, P)
    dq = np.ones((H, W), np.int32)
    dq.flat[rng.choice(P, P // 20, replace=False)] = 0
    with xg.Series(W, H, F, dpl, dq, dq, flatfield=flat, average=average) as s:
        s.ingest_sparse(nnz, idx, val)
        s.multitau(mode)
        got = s.g2ipif()
        assert s.info().float_path_pixels > P // 2
    rows, _ = oracle.sparse_filter(oracle.QMap(dq, dq), nnz, idx, val, F, average=average, flat=flat)
    want = oracle.multitau2(rows, F, dpl, mode)
    for g, w, which in zip(got, want, ("G2", "IP", "IF")):
        assert same_bits(g, w), (which, int(np.count_nonzero(g != w)))


@pytest.mark.parametrize("mode", [xg.MODE_REFERENCE, xg.MODE_EXACT])
@pytest.mark.parametrize("flat,dpl,average", [(False, 8, 1), (True, 4, 1), (False, 8, 2)])
def test_framesum_normalised_float_rows_vs_oracle(flat, dpl, average, mode):
    """normalize_by_framesum through the thread-per-pixel float kernel, with and
    without a flatfield and averaging, and rows past its capacity."""
    W, H, F = 310, 300, 150
    rng = np.random.default_rng(dpl + average)
    P, R = W * H, F * average
    hit = rng.random((R, P)) < rng.uniform(0.05, 0.15, (R, 1)) / average
    hit[:, :40] |= rng.random((R, 40)) < np.linspace(0.1, 1.0, 40)
    nnz, idx = hit.sum(1).astype(np.uint32), np.nonzero(hit)[1].astype(np.int32)
    val = rng.integers(1, 6, idx.size).astype(np.int16)
    gain = rng.uniform(0.8, 1.2, P) if flat else None
    dq = np.ones((H, W), np.int32)
    with xg.Series(W, H, F, dpl, dq, dq, flatfield=gain, average=average,
                   normalize_by_framesum=True) as s:
        s.ingest_sparse(nnz, idx, val)
        s.multitau(mode)
        got = s.g2ipif()
        assert s.info().float_path_pixels == P
    rows, side = oracle.sparse_filter(oracle.QMap(dq, dq), nnz, idx, val, F, average=average,
                                      flat=gain)
    want = oracle.multitau2(oracle.framesum_normalize(rows, side["frames_sum"], F), F, dpl, mode)
    for g, w, which in zip(got, want, ("G2", "IP", "IF")):
        assert same_bits(g, w), (which, int(np.count_nonzero(g != w)))
