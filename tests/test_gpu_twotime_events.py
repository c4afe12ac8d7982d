"""REFERENCE two-time from event lists and from the dense matrix, bit for bit
against the oracle: one frame, frame counts around the warp, the tile and the
columns per block, rows and columns of more than 32 events, and densities on
both sides of the rule that chooses between the two."""
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
