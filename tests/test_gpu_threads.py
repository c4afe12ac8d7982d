"""Distinct handles on distinct threads: two-time, multi-tau and float32
normalisation of series with different frame counts and delay schedules, whose
kernels ask for different amounts of shared memory, started over and over at
the same time.  Every call succeeds and gives the bits it gives alone."""
import threading

import numpy as np
import pytest

import xpcs_gpu as xg
from fixtures import same_bits_nan

pytestmark = pytest.mark.gpu

# side, frames, delays per level, mean counts
SERIES = [(40, 1600, 8, 0.02), (24, 90, 4, 0.05), (32, 700, 16, 0.02), (20, 60, 2, 0.03)]


def _work(s):
    out = [s.twotime([1, 2], static_map=True, window=3, mode=m)[k]
           for m in (xg.MODE_EXACT, xg.MODE_REFERENCE) for k in ("sg", "g2full", "g2partials")]
    s.multitau()
    return out + list(s.g2ipif()) + list(s.normalize())


def test_series_of_different_shapes_on_four_threads():
    series = []
    for k, (side, F, dpl, mean) in enumerate(SERIES):
        rng = np.random.default_rng(k)
        sq = (np.arange(side * side) * 4 // (side * side) + 1).astype(np.int32).reshape(side, side)
        s = xg.Series(side, side, F, dpl, (sq + 1) // 2, sq)
        hit = rng.random((F, side * side)) < mean
        idx = np.nonzero(hit)[1].astype(np.int32)
        s.ingest_sparse(hit.sum(1).astype(np.uint32), idx, np.ones(idx.size, np.int16))
        series.append(s)
    errors = []
    try:
        want = [_work(s) for s in series]
        start = threading.Barrier(len(series))

        def run(k):
            try:
                start.wait()
                for _ in range(60):
                    for a, b in zip(_work(series[k]), want[k]):
                        assert same_bits_nan(a, b)
            except Exception as e:  # reported below
                errors.append((SERIES[k], e))

        threads = [threading.Thread(target=run, args=(k,)) for k in range(len(series))]
        for t in threads:
            t.start()
        for t in threads:
            t.join()
        assert not errors, errors
    finally:
        for s in series:
            s.close()
