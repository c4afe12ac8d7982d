"""The filter's radix transpose over detector sizes at the edges of its digit
and pass counts (1 to 4 passes of 7 or 8 bits), both event tiles, with skipped
sub-frames (items that sort last), rows without events in long runs at the
start, in the middle and at the end, repeated (pixel, frame) events, and event
counts around a tile: the rows it makes against the oracle's, bit for bit."""
import numpy as np
import pytest

import oracle
import xpcs_gpu as xg
from fixtures import same_bits

pytestmark = pytest.mark.gpu

SIZES = [(3, 1), (9, 14), (127, 1), (16, 16), (113, 145), (128, 128), (181, 181), (256, 255),
         (256, 257), (1449, 1447), (2048, 1024), (2900, 1500), (4100, 4100)]


@pytest.mark.parametrize("tile", [8, 16])
@pytest.mark.parametrize("W,H", SIZES)
@pytest.mark.parametrize("events", [1, 2047, 2049, 20000])
def test_transposed_rows_vs_oracle(W, H, events, tile):
    if W * H > 5_000_000 and (events != 20000 or tile != 8):
        pytest.skip("one run of the largest detector")
    rng = np.random.default_rng(events + W)
    P, F, stride = W * H, 24, 2
    pix = rng.integers(P // 5, P - P // 7, events)
    pix[pix % 13 > 9] = P // 2  # a crowded pixel: repeated events too
    frame = np.sort(rng.integers(0, F * stride, events))
    nnz = np.bincount(frame, minlength=F * stride).astype(np.uint32)
    idx = pix.astype(np.int32)
    val = rng.integers(1, 4, events).astype(np.int16)
    dq = np.ones((H, W), np.int32)
    dq.flat[P // 3] = 0
    used = (frame % stride == 0) & (idx != P // 3)
    with xg.Series(W, H, F, 2, dq, dq, stride=stride) as s:
        s.set_tuning(radix_items_per_lane=tile)
        s.ingest_sparse(nnz, idx, val)
        s.multitau()
        if P > 5_000_000:  # the pixel sums alone
            want = np.bincount(idx[used], weights=val[used], minlength=P).astype(np.float32)
            ps, fs, _, _ = s.side_stats(max(F // 10, 1))
            assert same_bits(ps.ravel(), want / np.float32(F))
            return
        got = s.g2ipif()
        n = s.info().events
    rows, _ = oracle.sparse_filter(oracle.QMap(dq, dq), nnz, idx, val, F, stride=stride)
    assert n == rows.row_ptr[-1]
    want = oracle.multitau2(rows, F, 2, 0)
    for g, w, which in zip(got, want, ("G2", "IP", "IF")):
        assert same_bits(g, w), which
