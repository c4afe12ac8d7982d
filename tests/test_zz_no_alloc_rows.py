"""xpcs_multitau2_noalloc over every kind of row, bit for bit against the
oracle: lengths at the edges of the kernels that take them, integer and float
values, rows that are not regular (frames that repeat, descend or reach the
frame count, values that are not finite or too large to add) and schedules
with more delays in a level than a warp has lanes."""
import numpy as np
import pytest

import oracle
import xpcs_gpu as xg
from fixtures import same_bits_nan
from test_zz_no_alloc import _noalloc

pytestmark = pytest.mark.gpu

LENGTHS = [0, 1, 31, 32, 33, 79, 80, 81, 255, 256, 257, 1023, 1024, 1025, 4095, 4096, 4097, 4500]


def _case(F, lengths, seed):
    rng = np.random.default_rng(seed)
    rows = []
    for n in lengths:
        n = min(n, F)
        f = np.sort(rng.choice(F, n, replace=False)).astype(np.int32)
        ints = rng.integers(0, 3, n).astype(np.float32)
        rows.append((f, np.minimum(ints, 1.0) if n > 1500 else ints))  # sum below 4,096 or not
        rows.append((f, (rng.random(n) + 0.25).astype(np.float32)))
    return rows, rng


def _irregular(rows, rng, F):
    f = np.sort(rng.choice(F, 40, replace=False)).astype(np.int32)
    one = np.ones(40, np.float32)
    dup, down, past = f.copy(), f.copy(), f.copy()
    dup[11], down[20], past[-1] = dup[10], 0, F + 3
    inf, nan, huge = one.copy(), one.copy(), one.copy()
    inf[7], nan[9], huge[8:10] = np.inf, np.nan, 3e38
    return rows + [(dup, one), (down, one), (past, one), (f, inf), (f, nan), (f, huge)]


@pytest.mark.parametrize("F,dpl,spread", [
    (5000, 8, False), (5000, 4, True), (300, 16, True), (300, 20, True), (17000, 8, False),
    (70000, 4, False), (64, 4, True)])
@pytest.mark.parametrize("mode", [xg.MODE_REFERENCE, xg.MODE_EXACT])
def test_noalloc_rows_of_every_kind_vs_oracle(F, dpl, spread, mode):
    rows, rng = _case(F, LENGTHS, F + dpl)
    if spread:  # mostly short rows: the smaller row capacity
        rows += [(np.array([k % F], np.int32), np.ones(1, np.float32)) for k in range(4000)]
    rows = _irregular(rows, rng, F)
    rows = [rows[k] for k in rng.permutation(len(rows))]
    row_ptr = np.concatenate([[0], np.cumsum([r[0].size for r in rows])]).astype(np.int64)
    frame = np.concatenate([r[0] for r in rows])
    value = np.concatenate([r[1] for r in rows])
    got = _noalloc(row_ptr, frame, value, F, dpl, mode)
    want = oracle.multitau2(oracle.Rows(row_ptr, frame, value), F, dpl, mode)
    for name, g, w in zip(("G2", "IP", "IF"), got, want):
        assert same_bits_nan(g, w), (name, np.flatnonzero(
            ~((g == w) | (np.isnan(g) & np.isnan(w))).all(0)))
