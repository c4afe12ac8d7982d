"""REFERENCE two-time from event lists and from the dense matrix, bit for bit
against the oracle: one frame, frame counts around the warp, the tile and the
columns per block, rows and columns of more than 32 events, and densities on
both sides of the rule that chooses between the two."""
import time

import numpy as np
import pytest

import oracle
import xpcs_gpu as xg
from fixtures import same_bits_nan

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("W,H,F,density", [
    (9, 7, 1, 0.5), (12, 11, 8, 0.3), (40, 30, 33, 0.1), (13, 12, 65, 0.05), (13, 12, 65, 0.9),
    (10, 9, 300, 0.14), (10, 9, 300, 0.3), (16, 16, 130, 0.01), (5, 5, 3600, 0.02),
])
@pytest.mark.parametrize("static_map,average,threading", [(True, False, True), (False, True, False),
                                                          (True, True, False)])
def test_twotime_event_lists_and_dense_rows_vs_oracle(W, H, F, density, static_map, average,
                                                      threading):
    rng = np.random.default_rng(W * F)
    P = W * H
    sq = (rng.integers(0, 6, P) + 1).astype(np.int32)  # bins interleaved: mapping order matters
    sq[:12] = np.repeat(np.arange(1, 7), 2)  # every bin present, its second pixel too
    dq = (sq + 1) // 2
    hit = rng.random((F, P)) < density
    nnz, idx = hit.sum(1).astype(np.uint32), np.nonzero(hit)[1].astype(np.int32)
    val = rng.integers(1, 9, idx.size).astype(np.int16)
    dq, sq = dq.reshape(H, W), sq.reshape(H, W)
    qs, win = [1, 3], 3
    with xg.Series(W, H, F, 4, dq, sq) as s:
        s.ingest_sparse(nnz, idx, val)
        r = s.twotime(qs, static_map=static_map, average=average, window=win,
                      frame_threading=threading)
    qm = oracle.QMap(dq, sq)
    rows, _ = oracle.sparse_filter(qm, nnz, idx, val, F)
    o = oracle.twotime(qm, rows, F, qs, static_map, average, win, sort_pixels=threading)
    for q in qs:
        assert same_bits_nan(r["c2t"][q], o["c2t"][q])
    for k in ("sg", "g2full", "g2partials"):
        assert same_bits_nan(r[k], o[k]), k


@pytest.mark.parametrize("W,H,F,density,most", [
    (9, 7, 1, 0.04, 3), (12, 11, 8, 0.05, 9), (40, 30, 33, 0.03, 9), (13, 12, 65, 0.04, 2048),
    (30, 30, 900, 0.045, 4), (16, 16, 300, 0.02, 30000), (5, 5, 3600, 0.02, 9),
    (6, 5, 9500, 0.01, 9), (20, 20, 130, 0.3, 9),
])
@pytest.mark.parametrize("static_map,average", [(True, False), (False, True), (True, True),
                                                (False, False)])
def test_exact_twotime_from_event_lists_equals_the_int64_gram(W, H, F, density, most, static_map,
                                                              average):
    """EXACT mode from the event lists (one and several smoothing groups per q
    bin, columns of one and of many blocks, counts past what int32 or fp16 sums
    hold) equals the int64 CUDA-core Gram in every output."""
    rng = np.random.default_rng(W * F + most)
    P = W * H
    sq = (rng.integers(0, 6, P) + 1).astype(np.int32)
    sq[:12] = np.repeat(np.arange(1, 7), 2)
    dq = (sq + 1) // 2
    hit = rng.random((F, P)) < density
    nnz, idx = hit.sum(1).astype(np.uint32), np.nonzero(hit)[1].astype(np.int32)
    val = rng.integers(1, most + 1, idx.size).astype(np.int16)
    out = []
    for mode in (xg.MODE_EXACT, xg.TWOTIME_EXACT_CUDA_CORES):
        with xg.Series(W, H, F, 4, dq.reshape(H, W), sq.reshape(H, W)) as s:
            s.ingest_sparse(nnz, idx, val)
            out.append(s.twotime([1, 3], static_map=static_map, average=average, window=3,
                                 mode=mode))
    e, i = out
    for q in (1, 3):
        assert same_bits_nan(e["c2t"][q], i["c2t"][q])
    for k in ("sg", "g2full", "g2partials"):
        assert same_bits_nan(e[k], i[k]), k


@pytest.mark.parametrize("average", [False, True])
def test_exact_twotime_of_more_smoothing_groups_than_a_grid_has_rows(average):
    """68,644 static bins of one pixel each: with counts of 1, 2 and 4 every
    pixel's smoothed pair of events is 1 to the bit (or, averaged over the
    frames, its counts over their mean), and C is their number over the pixels."""
    W = H = 262
    P, F = W * H, 6
    rng = np.random.default_rng(3)
    sq = np.arange(1, P + 1, dtype=np.int32).reshape(H, W)
    v = np.where(rng.random((F, P)) < 0.04, 2 ** rng.integers(0, 3, (F, P)), 0)
    hit = v > 0
    nnz, idx = hit.sum(1).astype(np.uint32), np.nonzero(hit)[1].astype(np.int32)
    with xg.Series(W, H, F, 4, np.ones((H, W), np.int32), sq) as s:
        s.ingest_sparse(nnz, idx, v[hit].astype(np.int16))
        r = s.twotime([1], static_map=True, average=average, mode=xg.MODE_EXACT)
    want = np.zeros((F, F))
    sg = v.mean(0) if average else None
    for a in range(F):
        for b in range(a, F):
            both = hit[a] & hit[b]
            w = (v[a] * v[b])[both] / sg[both] ** 2 if average else np.ones(np.count_nonzero(both))
            want[a, b] = w.sum() / P
    assert np.allclose(r["c2t"][1], want, rtol=2.0 ** -23, atol=0)
    assert np.array_equal(r["sg"], v.mean(0).astype(np.float32)[:, None] if average
                          else v.T.astype(np.float32))


def _bright_ring(W, H, F, ring, density, seed=0):
    """A q bin of `ring` pixels hit in `density` of the frames on a detector that
    is dark elsewhere."""
    rng = np.random.default_rng(seed)
    P = W * H
    dq = np.full(P, 2, np.int32)
    dq[rng.choice(P - 2, ring, replace=False) + 1] = 1
    hit = rng.random((F, P)) < np.where(dq == 1, density, 0.002)
    nnz, idx = hit.sum(1).astype(np.uint32), np.nonzero(hit)[1].astype(np.int32)
    return dq.reshape(H, W), nnz, idx, rng.integers(1, 5, idx.size).astype(np.int16)


def test_a_bright_ring_alone_takes_the_dense_forms():
    """The lists' work is in pairs of events of the processed rows, whatever the
    rest of the detector holds: EXACT mode runs the tensor-core Gram (it reports
    its time), with the int64 Gram's bits, and REFERENCE mode the tiled Gram: it
    takes about as long as with the same rows dense enough by themselves."""
    W, H, F, ring = 200, 180, 700, 1500
    dq, nnz, idx, val = _bright_ring(W, H, F, ring, 0.9)
    keep = dq.ravel()[idx] == 1
    alone = (np.bincount(np.repeat(np.arange(F), nnz)[keep], minlength=F).astype(np.uint32),
             idx[keep], val[keep])
    only = np.where(dq == 1, 1, 0).astype(np.int32)
    out = {}
    for name, m, frames in (("all", dq, (nnz, idx, val)), ("only", only, alone)):
        with xg.Series(W, H, F, 4, m, m) as s:
            s.ingest_sparse(*frames)
            for mode in (xg.MODE_REFERENCE, xg.MODE_EXACT, xg.TWOTIME_EXACT_CUDA_CORES):
                ms = []
                for _ in range(4):
                    t = time.perf_counter()
                    r = s.twotime([1], window=3, mode=mode)
                    ms.append(time.perf_counter() - t)
                out[name, mode] = r, min(ms)
    for mode in (xg.MODE_REFERENCE, xg.MODE_EXACT, xg.TWOTIME_EXACT_CUDA_CORES):
        a, o = out["all", mode], out["only", mode]
        assert same_bits_nan(a[0]["c2t"][1], o[0]["c2t"][1])
        if mode == xg.MODE_REFERENCE:
            assert a[1] < 2 * o[1] + 1e-3, (a[1], o[1])
    assert out["all", xg.MODE_EXACT][0]["gram_ms"] > 0
    assert same_bits_nan(out["all", xg.MODE_EXACT][0]["c2t"][1],
                         out["all", xg.TWOTIME_EXACT_CUDA_CORES][0]["c2t"][1])


@pytest.mark.parametrize("threading", [False, True])
def test_a_bright_ring_in_the_reference_order_vs_oracle(threading):
    W, H, F = 40, 36, 90
    dq, nnz, idx, val = _bright_ring(W, H, F, 60, 0.95, seed=2)
    with xg.Series(W, H, F, 4, dq, dq) as s:
        s.ingest_sparse(nnz, idx, val)
        for qs in ([1], [2], [1, 2]):
            r = s.twotime(qs, static_map=True, window=3, frame_threading=threading)
            qm = oracle.QMap(dq, dq)
            rows, _ = oracle.sparse_filter(qm, nnz, idx, val, F)
            o = oracle.twotime(qm, rows, F, qs, True, False, 3, sort_pixels=threading)
            for q in qs:
                assert same_bits_nan(r["c2t"][q], o["c2t"][q])
            for k in ("sg", "g2full", "g2partials"):
                assert same_bits_nan(r[k], o[k]), k
