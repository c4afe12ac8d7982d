"""xpcs_multitau2 with as many pixels as give every short row a thread: row
lengths at the edges of the kernels' capacities, integer and float values, bit
for bit against the oracle."""
import numpy as np
import pytest

import oracle
import xpcs_gpu as xg
from fixtures import same_bits

pytestmark = pytest.mark.gpu

EDGES = [0, 1, 31, 32, 33, 48, 49, 64, 65, 80, 81, 112, 113, 255, 256, 257, 1023, 1024, 1025]


@pytest.mark.parametrize("pixels,F,dpl,mean", [(33003, 2000, 8, 4), (33003, 1200, 4, 40),
                                               (5001, 2000, 16, 20)])
@pytest.mark.parametrize("mode", [xg.MODE_REFERENCE, xg.MODE_EXACT])
def test_caller_held_rows_of_many_pixels_vs_oracle(pixels, F, dpl, mean, mode):
    rng = np.random.default_rng(pixels + F)
    n = np.minimum(rng.poisson(mean, pixels), F)
    n[rng.choice(pixels, len(EDGES), replace=False)] = EDGES
    frame = [np.sort(rng.choice(F, k, replace=False)) for k in n]
    row_ptr = np.concatenate([[0], np.cumsum(n)]).astype(np.int64)
    frame = np.concatenate(frame).astype(np.int32)
    value = rng.integers(1, 4, frame.size).astype(np.float32)
    for p in range(0, pixels, 97):  # float rows
        value[row_ptr[p]:row_ptr[p + 1]] += 0.25
    got = xg.multitau2(row_ptr, frame, value, F, dpl, mode)
    want = oracle.multitau2(oracle.Rows(row_ptr, frame, value), F, dpl, mode)
    for g, w, which in zip(got, want, ("G2", "IP", "IF")):
        assert same_bits(g, w), which
