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


SPAN = 4096  # rows of a gap that a warp fills
AROUND = [k * SPAN + d for k in (1, 2, 3, 9, 36) for d in (-2, -1, 0, 1)]


@pytest.mark.parametrize("pixels", [
    [0], [153599], [0, 153599], AROUND, AROUND[::2], AROUND[1::3], [5 * SPAN], [5 * SPAN - 1],
    [5 * SPAN, 6 * SPAN], [5 * SPAN - 1, 6 * SPAN - 1], [5 * SPAN, 6 * SPAN - 1], list(range(153600)),
])
def test_row_pointers_across_gaps_of_whole_spans(pixels):
    """Rows without events between events at the edges of the spans that warps of
    their own fill, and no event kept at all (the skipped sub-frames')."""
    W, H, F = 480, 320, 8
    P = W * H
    dq = np.ones((H, W), np.int32)
    for kept in (True, False):
        nnz = np.zeros(2 * F, np.uint32)
        nnz[[4, 10] if kept else [5, 11]] = len(pixels)
        idx = np.array(pixels * 2, np.int32)
        val = np.arange(1, idx.size + 1).astype(np.int16) % 7 + 1
        with xg.Series(W, H, F, 2, dq, dq, stride=2) as s:
            s.ingest_sparse(nnz, idx, val)
            s.multitau()
            got = s.g2ipif()
            assert s.info().events == (idx.size if kept else 0)
        rows, _ = oracle.sparse_filter(oracle.QMap(dq, dq), nnz, idx, val, F, stride=2)
        for g, w, which in zip(got, oracle.multitau2(rows, F, 2, 0), ("G2", "IP", "IF")):
            assert same_bits(g, w), (which, kept)


def test_a_large_detectors_events_in_one_corner_take_no_longer():
    """16.8 M pixels: the filter of 20,000 events in one corner, or of none that
    is kept, takes about as long as that of events all over the detector."""
    W = H = 4096
    P, F, n = W * H, 8, 20000
    rng = np.random.default_rng(1)
    dq = np.ones((H, W), np.int32)
    ms = {}
    with xg.Series(W, H, F, 1, dq, dq, stride=2) as s:
        for name, last, frame in (("all over", P, 4), ("corner", 30000, 4), ("none", P, 5)):
            nnz = np.zeros(2 * F, np.uint32)
            nnz[frame] = n
            idx = np.sort(rng.choice(last, n, replace=False)).astype(np.int32)
            s.reset()
            s.ingest_sparse(nnz, idx, np.ones(n, np.int16))
            t = []
            for _ in range(6):
                s.multitau()
                s.synchronize()
                t.append(s.stage_times()["filter_ms"])
            ms[name] = min(t)
    assert ms["corner"] < 1.5 * ms["all over"] and ms["none"] < 1.5 * ms["all over"], ms
