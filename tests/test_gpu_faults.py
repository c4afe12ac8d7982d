"""Failures injected on the host, checked on the GPU without faulting it: an
allocation refused by the library's device-memory limit must come back as
XPCS_ERR_OUT_OF_MEMORY, leave the handle usable, and leak nothing; a sparse
frame with a pixel index outside the detector must come back as
XPCS_ERR_INPUT (the reference would write out of bounds,
sparse_filter.cpp:168-187)."""
import numpy as np
import pytest

import xpcs_gpu as xg
from fixtures import load, same_bits

pytestmark = pytest.mark.gpu


def _series(fx):
    return xg.Series(fx["W"], fx["H"], fx["F"], fx["dpl"], fx["dqmap"], fx["sqmap"],
                     static_window=fx["swin"], device=0)


def test_device_memory_limit_refuses_cleanly_and_the_handle_recovers():
    fx = load("sparse_basic")
    used0, _ = xg.device_memory(0)
    try:
        with _series(fx) as s:
            s.ingest_sparse(fx["nnz"], fx["idx"], fx["val"])
            s.synchronize()
            used1, _ = xg.device_memory(0)
            assert used1 > used0
            # room for a few bytes more than the series holds: the transpose needs more
            xg.set_device_memory_limit(0, used1 + 64)
            with pytest.raises(xg.XpcsError) as e:
                s.multitau(xg.MODE_REFERENCE)
            assert e.value.code == 3 and "limit" in str(e.value)
            assert xg.device_memory(0)[0] <= used1 + 64
            xg.set_device_memory_limit(0, 0)
            s.multitau(xg.MODE_REFERENCE)
            G2, IP, IF = s.g2ipif()
        for name, got in (("G2", G2), ("IP", IP), ("IF", IF)):
            assert same_bits(got, fx["ref_" + name]), name
    finally:
        xg.set_device_memory_limit(0, 0)
    assert xg.device_memory(0)[0] == used0  # everything the series held was returned


def test_series_creation_over_the_limit_is_refused():
    fx = load("sparse_basic")
    used0, _ = xg.device_memory(0)
    try:
        xg.set_device_memory_limit(0, used0 + 16)
        with pytest.raises(xg.XpcsError) as e:
            _series(fx)
        assert e.value.code == 3
    finally:
        xg.set_device_memory_limit(0, 0)
    assert xg.device_memory(0)[0] == used0


def test_pixel_index_outside_the_detector_is_an_input_error():
    fx = load("sparse_basic")
    idx = fx["idx"].copy()
    idx[len(idx) // 2] = fx["W"] * fx["H"] + 7
    with _series(fx) as s:
        s.ingest_sparse(fx["nnz"], idx, fx["val"])
        s.multitau(xg.MODE_REFERENCE)
        with pytest.raises(xg.XpcsError) as e:
            s.synchronize()
        assert e.value.code == 6
        # the same handle, reset and given good frames, gives the reference's result
        s.reset()
        s.ingest_sparse(fx["nnz"], fx["idx"], fx["val"])
        s.multitau(xg.MODE_REFERENCE)
        G2 = s.g2ipif()[0]
    assert same_bits(G2, fx["ref_G2"])
    assert np.all(np.isfinite(G2))


def test_device_properties_and_bad_ordinal():
    assert xg.device_sm_count(0) >= 1
    with pytest.raises(xg.XpcsError) as e:
        xg.device_sm_count(1 << 20)
    assert e.value.code == 1


@pytest.mark.parametrize("mode,side,F,density,need", [
    # REFERENCE: the dense rows [P][F]; EXACT: X^T of a group and F x F matrices
    (xg.MODE_REFERENCE, 200, 100, 0.39, lambda P, F: 4 * P * F),
    (xg.MODE_EXACT, 20, 900, 0.04, lambda P, F: 20 * F * F + (8 << 20)),
    (xg.MODE_EXACT, 300, 100, 0.05, lambda P, F: 2 * 128 * P // 6 + 20 * F * F + (1 << 19)),
])
def test_two_time_within_what_a_limit_left_it_before(mode, side, F, density, need):
    """Event lists are no condition of a two-time call: a limit that leaves room
    for the dense forms and the results is enough."""
    rng = np.random.default_rng(F)
    P = side * side
    sq = (np.arange(P) * 6 // P + 1).astype(np.int32).reshape(side, side)
    hit = rng.random((F, P)) < density
    nnz, idx = hit.sum(1).astype(np.uint32), np.nonzero(hit)[1].astype(np.int32)
    try:
        out = []
        for limit in (False, True):
            with xg.Series(side, side, F, 2, sq, sq) as s:
                s.ingest_sparse(nnz, idx, np.ones(idx.size, np.int16))
                s.multitau()
                s.synchronize()
                if limit:
                    xg.set_device_memory_limit(0, xg.device_memory(0)[0] + 16 * P + 4 * 7 * F * F
                                               + need(P, F) + (1 << 20))
                out.append(s.twotime(range(1, 7), window=2, mode=mode))
        a, b = out
        for q in range(1, 7):
            assert same_bits(a["c2t"][q], b["c2t"][q])
        for k in ("sg", "g2full", "g2partials"):
            assert same_bits(a[k], b[k]), k
    finally:
        xg.set_device_memory_limit(0, 0)


def _flat_series(F=300):
    W, H = 310, 300
    rng = np.random.default_rng(5)
    n = rng.poisson(0.04, (F, W * H))
    hit = n > 0
    nnz, idx, val = hit.sum(1).astype(np.uint32), np.nonzero(hit)[1], n[hit]
    dq = np.ones((H, W), np.int32)
    s = xg.Series(W, H, F, 8, dq, dq, flatfield=rng.uniform(0.8, 1.2, W * H))
    s.ingest_sparse(nnz, idx.astype(np.int32), val.astype(np.int16))
    s.synchronize()
    return s, idx.size


def test_float_rows_within_what_a_limit_left_them_before():
    """The scratch of the thread-per-pixel float kernel (as large as G2, IP and
    IF, and its rows' slots) is no condition of a call: a limit that leaves room
    for the event lists (54 B per event), the per-pixel tables and the results
    is enough, alone and in a batch; what a call did take of it is given back."""
    try:
        s, events = _flat_series()
        with s:
            s.multitau(xg.MODE_REFERENCE)
            want = s.g2ipif()
            assert s.info().float_path_pixels > s.P // 2
            room = s.P * (12 * s.D + 64) + 54 * events + (4 << 20)
        for limited_room in (room, 1 << 34):
            s, _ = _flat_series()
            with s:
                xg.set_device_memory_limit(0, xg.device_memory(0)[0] + limited_room)
                for _ in range(2):
                    s.multitau(xg.MODE_REFERENCE)
                    for g, w in zip(s.g2ipif(), want):
                        assert same_bits(g, w)
                    assert s.info().float_path_pixels > s.P // 2
                    s.normalize(f32=False)
                with xg.Batch([s]) as b:
                    for queue in (True, False):
                        b.set_form(queue)
                        for k in range(3):
                            b.run(f64=False)
                            for g, w in zip(s.g2ipif(), want):
                                assert same_bits(g, w)
                            if k == 1:
                                s.multitau(xg.MODE_REFERENCE)
                assert xg.device_memory(0)[0] < xg.device_memory(0)[1] - limited_room + room
                xg.set_device_memory_limit(0, 0)
                b = xg.Batch([s])
                b.run(f64=False)
                b.run(f64=False)  # captured with the scratch, which the next call gives back
                xg.set_device_memory_limit(0, xg.device_memory(0)[0] + limited_room)
                s.multitau(xg.MODE_REFERENCE)
                b.run(f64=False)
                for g, w in zip(s.g2ipif(), want):
                    assert same_bits(g, w)
                b.close()
                xg.set_device_memory_limit(0, 0)
    finally:
        xg.set_device_memory_limit(0, 0)


def test_blocks_joined_within_what_a_limit_left_them_before():
    """The places of the blocks' rows (4 B per pixel and block) are no condition
    of the join: 260 blocks of one frame under a limit that leaves room for the
    event lists and the results."""
    W, H, F = 300, 290, 260
    rng = np.random.default_rng(8)
    n = rng.poisson(0.01, (F, W * H))
    hit = n > 0
    nnz, idx, val = hit.sum(1).astype(np.uint32), np.nonzero(hit)[1], n[hit]
    dq = np.ones((H, W), np.int32)
    try:
        out = []
        for block in (0, 1):
            with xg.Series(W, H, F, 4, dq, dq) as s:
                s.set_block_frames(block)
                s.ingest_sparse(nnz, idx.astype(np.int32), val.astype(np.int16))
                s.synchronize()
                used = xg.device_memory(0)[0]
                if block:
                    xg.set_device_memory_limit(0, used + s.P * (12 * s.D + 64) + 54 * idx.size
                                               + (4 << 20))
                for _ in range(2):
                    s.multitau(xg.MODE_REFERENCE)
                    out.append(s.g2ipif())
        for r in out[1:]:
            for g, w in zip(r, out[0]):
                assert same_bits(g, w)
    finally:
        xg.set_device_memory_limit(0, 0)


def test_counts_too_large_for_the_lists_within_what_the_int64_gram_takes():
    """EXACT two-time that first looks at the counts' lists and then takes the
    int64 Gram needs no more than asking for that Gram does."""
    side, F = 300, 100
    rng = np.random.default_rng(4)
    P = side * side
    sq = (np.arange(P) * 2 // P + 1).astype(np.int32).reshape(side, side)
    hit = rng.random((F, P)) < 0.02
    nnz, idx = hit.sum(1).astype(np.uint32), np.nonzero(hit)[1].astype(np.int32)
    val = rng.integers(1, 30000, idx.size).astype(np.int16)
    try:
        out, need = [], 0
        for mode in (xg.TWOTIME_EXACT_CUDA_CORES, xg.MODE_EXACT):
            with xg.Series(side, side, F, 2, sq, sq) as s:
                s.ingest_sparse(nnz, idx, val)
                s.multitau()
                s.synchronize()
                used = xg.device_memory(0)[0]
                xg.set_device_memory_limit(0, used + (need + 4096 if need else 1 << 34))
                out.append(s.twotime([1, 2], window=2, mode=mode))
                need = xg.device_memory(0)[0] - used
                xg.set_device_memory_limit(0, 0)
        for q in (1, 2):
            assert same_bits(out[0]["c2t"][q], out[1]["c2t"][q])
    finally:
        xg.set_device_memory_limit(0, 0)
