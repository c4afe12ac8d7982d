"""stderr in float64 of q rings whose ratios lie close together or whose first
pixels are dark, where sums about a shift cancel: one pixel, equal rows, dead
pixels first (within one chunk of pixels and in the first of several).

Tolerances: a ratio is good to a few 2^-48, so equal ratios deviate from their
mean by at most a few 2^-48 of it, and the spread of the others here, some
percent of the ratio, is good to about 2^-48 x 50 relative, below 1e-12."""
import numpy as np
import pytest

import oracle
import xpcs_gpu as xg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("frames,dpl", [(64, 4), (257, 8)])
def test_stderr_of_rings_with_little_spread_or_dead_pixels(frames, dpl):
    rng = np.random.default_rng(frames)
    H, W = 30, 40
    P = H * W
    dq = np.zeros(P, np.int32)
    lam = np.zeros(P)
    ones = list(range(1, 41))  # 40 rings of one pixel
    dq[:40] = ones
    lam[:40] = 8.0
    dq[40:100], lam[40:100] = 41, 8.0          # 60 equal rows
    dq[100:200], lam[100 + 32:200] = 42, 12.0  # one chunk, its first 32 pixels dark
    dq[200:900], lam[300:900] = 43, 12.0       # several chunks, the first ratios 0
    dq[900:1200], lam[900:1200] = 44, 12.0     # an ordinary ring
    counts = rng.poisson(lam, (frames, P)).astype(np.int16)
    counts[:, 40:100] = counts[:, 40:41]
    counts = np.minimum(counts, 4000 // frames)  # integer rows
    hit = counts != 0
    nnz, idx = hit.sum(1).astype(np.uint32), np.nonzero(hit)[1].astype(np.int32)
    val = counts[hit]
    dq = dq.reshape(H, W)
    with xg.Series(W, H, frames, dpl, dq, dq) as s:
        s.ingest_sparse(nnz, idx, val)
        s.multitau()
        G2, IP, IF = s.g2ipif()
        g2, se, _, _ = s.normalize(f32=False)
    og2, ose = oracle.normalize_f64(oracle.QMap(dq, dq), G2, IP, IF)
    assert np.allclose(g2, og2, rtol=1e-12, atol=0)
    assert np.all(se[:, :40] == 0.0), se[:, :40]
    assert np.all(se[:, 40] <= 2.0 ** -44 * og2[:, 40]), se[:, 40]
    assert np.allclose(se[:, 41:], ose[:, 41:], rtol=1e-12, atol=0)
