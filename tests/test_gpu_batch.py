"""Batches (xpcs_batch_*): several series of uneven shapes run as one CUDA
graph.  Each member's G2/IP/IF and g2/stderr (float64 and float32) must be
bit-identical to the same series run alone, the graph replay must repeat
them, a member whose frames change must be recaptured, and golden members
must still match the reference's own outputs."""
import time

import numpy as np
import pytest

import xpcs_gpu as xg
import xpcs_synth as xs
from fixtures import load, same_bits, same_bits_nan

pytestmark = pytest.mark.gpu

# uneven members: detector side, frames, mean photons/pixel/frame, delays per level, tau range
MIX = [(64, 300, 0.02, 4, (2, 50)), (96, 1500, 0.004, 8, (5, 300)), (48, 4000, 0.01, 8, (10, 900)),
       (128, 600, 0.05, 4, (2, 20)), (80, 2500, 0.03, 8, (20, 2000)), (40, 200, 0.2, 4, (2, 10))]


def synth_member(i, side, F, mean, dpl, tau, seed_shift=0):
    acq = xs.Acquisition(width=side, height=side, frames=F, n_static=12, n_dynamic=6, mean=mean,
                         tau_min=tau[0], tau_max=tau[1], seed=100 + i + seed_shift, dpl=dpl)
    dq, sq, _, _ = xs.maps(acq)
    nnz, idx, val = xs.sparse_frames(acq)
    return acq, dq, sq, (nnz, idx, val)


def open_member(acq, dq, sq, frames):
    s = xg.Series(acq.width, acq.height, acq.frames, acq.dpl, dq, sq)
    s.ingest_sparse(*frames)
    return s


def golden_member(name):
    fx = load(name)
    if fx["dense"]:
        nd = fx["ndark"]
        s = xg.Series(fx["W"], fx["H"], fx["F"], fx["dpl"], fx["dqmap"], fx["sqmap"],
                      flatfield=fx["flatfield"], static_window=fx["swin"], dense=True,
                      lld=float(fx["lld_sigma"][0]), sigma=float(fx["lld_sigma"][1]))
        s.set_dark(fx["raw"][:nd])
        s.ingest_dense(fx["raw"][nd:])
    else:
        s = xg.Series(fx["W"], fx["H"], fx["F"], fx["dpl"], fx["dqmap"], fx["sqmap"],
                      flatfield=fx["flatfield"], stride=fx["stride"], average=fx["avg"],
                      static_window=fx["swin"])
        s.ingest_sparse(fx["nnz"], fx["idx"], fx["val"])
    return fx, s


def results(s, f32=True):
    G2, IP, IF = s.g2ipif()
    g64, s64, g32, s32 = s.normalized(f64=True, f32=f32)
    return dict(G2=G2, IP=IP, IF=IF, g64=g64, s64=s64, g32=g32, s32=s32)


def alone(s, mode):
    s.multitau(mode)
    s.normalize()
    return results(s)


def assert_same(a, b):
    for k in ("G2", "IP", "IF"):
        assert same_bits(a[k], b[k]), k
    for k in ("g64", "s64", "g32", "s32"):
        if a[k] is not None and b[k] is not None:
            assert same_bits_nan(a[k], b[k]), k


@pytest.mark.parametrize("mode", [xg.MODE_REFERENCE, xg.MODE_EXACT])
def test_batch_equals_each_series_alone(mode):
    members = [open_member(*synth_member(i, *m)) for i, m in enumerate(MIX)]
    goldens = [golden_member(n) for n in ("sparse_quirk", "sparse_stride_avg", "dense_dark")]
    series = members + [s for _, s in goldens]
    try:
        solo = [alone(s, mode) for s in series]
        with xg.Batch(series) as b:
            b.run(mode, f64=True, f32=True)
            ms, kernels, _ = b.stats()
            assert ms > 0 and kernels >= 10 * len(series)
            for s, r in zip(series, solo):
                assert_same(results(s), r)
            b.run(mode, f64=True, f32=True)  # graph replay
            for s, r in zip(series, solo):
                assert_same(results(s), r)
        if mode == xg.MODE_REFERENCE:
            for fx, s in goldens:
                r = results(s)
                for k in ("G2", "IP", "IF"):
                    assert same_bits(r[k], fx["ref_" + k]), k
                assert same_bits_nan(r["g32"], fx["ref_norm_0_g2"])
                assert same_bits_nan(r["s32"], fx["ref_norm_0_stderr"])
    finally:
        for s in series:
            s.close()


def test_batch_recaptures_when_a_member_changes():
    built = [synth_member(i, *m) for i, m in enumerate(MIX[:3])]
    series = [open_member(a, d, q, f) for a, d, q, f in built]
    try:
        with xg.Batch(series) as b:
            b.run()
            first = [results(s, f32=False) for s in series]
            # new frames for member 1 (same maps): the batch must notice and capture again
            _, _, _, frames = synth_member(1, *MIX[1], seed_shift=50)
            acq, dq, sq, _ = built[1]
            series[1].reset()
            series[1].ingest_sparse(*frames)
            b.run()
            changed = results(series[1], f32=False)
            assert not same_bits(changed["G2"], first[1]["G2"])
            for k in (0, 2):
                assert_same(results(series[k], f32=False), first[k])
            with open_member(acq, dq, sq, frames) as ref:
                r = alone(ref, xg.MODE_REFERENCE)
            for k in ("G2", "IP", "IF", "g64", "s64"):
                assert same_bits_nan(changed[k], r[k]), k
            # float32 normalisation was not requested in this run
            with pytest.raises(xg.XpcsError):
                series[0].normalized(f64=False, f32=True)
    finally:
        for s in series:
            s.close()


def test_autotune_changes_time_not_results():
    series = [open_member(*synth_member(i, *m)) for i, m in enumerate(MIX[:4])]
    try:
        before = [alone(s, xg.MODE_REFERENCE) for s in series]
        caps = [s.autotune() for s in series]
        assert all(c in (32, 48, 64, 80, 112) for c in caps)
        for s, r in zip(series, before):
            assert_same(alone(s, xg.MODE_REFERENCE), r)
        fresh = [open_member(*synth_member(i, *m)) for i, m in enumerate(MIX[4:], start=4)]
        solo = [alone(s, xg.MODE_REFERENCE) for s in fresh]
        with xg.Batch(series + fresh) as b:
            b.run(autotune=True, f32=True)
            for s, r in zip(series + fresh, before + solo):
                assert_same(results(s), r)
        for s in fresh:
            s.close()
    finally:
        for s in series:
            s.close()


def test_framesum_series_cannot_join_a_batch():
    fx, s = golden_member("sparse_quirk")
    fs = xg.Series(fx["W"], fx["H"], fx["F"], fx["dpl"], fx["dqmap"], fx["sqmap"],
                   normalize_by_framesum=True)
    try:
        with pytest.raises(xg.XpcsError):
            xg.Batch([s, fs])
    finally:
        s.close()
        fs.close()


def test_batch_timeline_covers_every_member():
    data = [synth_member(i, *m) for i, m in enumerate(MIX)]
    series = [open_member(*d) for d in data]
    try:
        b = xg.Batch(series)
        with pytest.raises(xg.XpcsError):
            b.timeline()  # not run yet
        b.run(xg.MODE_REFERENCE, f64=True)
        start, end = b.timeline()
        ms = b.stats()[0]
        assert start.shape == (len(series),) and np.all(start >= 0) and np.all(end > start)
        # every member's work lies inside the graph's run (timer resolution slack)
        assert float(np.max(end)) <= ms + 0.05
        b.close()
    finally:
        for s in series:
            s.close()


@pytest.mark.parametrize("mode", [xg.MODE_REFERENCE, xg.MODE_EXACT])
def test_every_knob_setting_gives_the_same_bits(mode):
    """Row capacity (warps per pixel), scratch words (level-fold schedule) and
    transpose tile change the work, never the results; bad values are refused."""
    members = [synth_member(i, *m) for i, m in enumerate(MIX[:3])]
    for acq, dq, sq, frames in members:
        s = open_member(acq, dq, sq, frames)
        try:
            ref = alone(s, mode)
            for cap, extra, ipt in ((32, 0, 8), (48, 8, 16), (64, 8, 0), (112, 0, 16),
                                    (80, 8, 8)):
                s.set_tuning(cap, extra, ipt)
                assert s.tuning() == {"thread_cap": cap, "scratch_extra": extra,
                                      "radix_items_per_lane": ipt}
                assert_same(alone(s, mode), ref)
            s.autotune(mode)
            t = s.tuning()
            assert t["thread_cap"] in (32, 48, 64, 80, 112) and t["scratch_extra"] in (0, 8)
            assert t["radix_items_per_lane"] in (8, 16)
            assert_same(alone(s, mode), ref)
            for bad in ((40, 0, 0), (80, 4, 0), (80, 0, 12)):
                with pytest.raises(xg.XpcsError):
                    s.set_tuning(*bad)
        finally:
            s.close()


LONG_ROWS = [(48, 4000, 0.15, 8, (10, 300)), (24, 8000, 0.25, 8, (5, 800))]


@pytest.mark.parametrize("queue", [True, False])
def test_both_batch_forms_equal_each_series_alone(queue):
    """The work-queue form (multi-tau of every member as persistent launches
    pulling 32-pixel groups and rows from device counters) and the chains form
    give each member the bits it gets alone: rows of every kernel class, from
    short thread-per-pixel rows to 1,000-4,000-event warp-per-pixel rows and
    float rows (flatfield, dense)."""
    members = [open_member(*synth_member(i, *m)) for i, m in enumerate(MIX + LONG_ROWS)]
    goldens = [golden_member(n) for n in ("sparse_flat", "dense_dark")]
    series = members + [s for _, s in goldens]
    try:
        solo = [alone(s, xg.MODE_REFERENCE) for s in series]
        with xg.Batch(series) as b:
            b.set_form(queue)
            b.run(xg.MODE_REFERENCE, f64=True, f32=True)
            assert b.form() == (queue, len(series))
            for s, r in zip(series, solo):
                assert_same(results(s), r)
            b.run(xg.MODE_REFERENCE, f64=True, f32=True, autotune=True)
            assert b.form()[0] == queue  # autotuning keeps the chosen form
            for s, r in zip(series, solo):
                assert_same(results(s), r)
            start, end = b.timeline()
            assert np.all(end > start)
    finally:
        for s in series:
            s.close()


def test_first_run_replay_and_a_change_of_form_give_the_same_bits():
    """The first run on new frames enqueues the members' work directly, the
    next ones replay a captured graph; a form chosen in between, and calls on
    a member alone, leave the results as they are."""
    series = [open_member(*synth_member(i, *m)) for i, m in enumerate(MIX[:4])]
    golden = [golden_member(n)[1] for n in ("sparse_flat", "dense_dark")]
    members = series + golden
    try:
        solo = [alone(s, xg.MODE_REFERENCE) for s in members]
        with xg.Batch(members) as b:
            for queue in (True, True, False, False, True):
                b.set_form(queue)
                for _ in range(3):
                    b.run(xg.MODE_REFERENCE, f64=True, f32=True)
                    for s, r in zip(members, solo):
                        assert_same(results(s), r)
                    members[1].side_stats(max(members[1].frames // 10, 1))
            b.run(xg.MODE_EXACT, f64=True)
            b.run(xg.MODE_REFERENCE, f64=True, f32=True)
            for s, r in zip(members, solo):
                assert_same(results(s), r)
    finally:
        for s in members:
            s.close()


@pytest.mark.parametrize("queue", [True, False])
def test_a_member_run_alone_in_another_mode_leaves_the_batch_its_results(queue):
    """A member run alone in the other mode holds that mode's plan: the batch
    puts its own back before its graph is captured and before each replay."""
    series = [open_member(*synth_member(i, *m)) for i, m in enumerate(MIX[:4])]
    series.append(open_member(*synth_member(0, *LONG_ROWS[0])))
    other = {xg.MODE_REFERENCE: xg.MODE_EXACT, xg.MODE_EXACT: xg.MODE_REFERENCE}
    try:
        solo = {m: [alone(s, m) for s in series] for m in other}
        assert any(not same_bits(a["G2"], b["G2"]) for a, b in zip(*solo.values()))
        with xg.Batch(series) as b:
            b.set_form(queue)
            for mode in other:
                for _ in range(3):  # enqueued directly, captured, replayed
                    b.run(mode, f64=True, f32=True)
                    for s, r in zip(series, solo[mode]):
                        assert_same(results(s), r)
                    for s in series:
                        s.multitau(other[mode])
                        s.synchronize()
    finally:
        for s in series:
            s.close()


def test_a_replay_waits_for_what_a_member_was_asked_alone():
    """xpcs_multitau returns with its work enqueued on the member's stream: the
    batch's graph, captured or replayed, starts after it."""
    series = [open_member(*synth_member(i, *m)) for i, m in enumerate(MIX[1:] + LONG_ROWS)]
    try:
        solo = [alone(s, xg.MODE_REFERENCE) for s in series]
        with xg.Batch(series) as b:
            for _ in range(6):
                b.run(xg.MODE_REFERENCE, f64=True, f32=True)
                for s, r in zip(series, solo):
                    assert_same(results(s), r)
                for s in series:
                    s.multitau(xg.MODE_REFERENCE)
    finally:
        for s in series:
            s.close()


def test_autotuning_after_a_change_of_form_times_the_chain_counts_again():
    """A form chosen on frames that the batch has run leaves the chain count to
    the next autotuned run: that run captures one graph for each of 1, 2, 4 and
    8 chains and the one it keeps, where a run without autotuning captures one."""
    series = [open_member(*synth_member(i, *m)) for i, m in enumerate(MIX + LONG_ROWS)]
    took = {}
    try:
        solo = [alone(s, xg.MODE_REFERENCE) for s in series]
        for tune in (False, True):
            with xg.Batch(series) as b:
                b.run(autotune=tune, f32=True)
                b.run(autotune=tune, f32=True)
                ms = []
                for queue in (True, False) * 3:
                    b.set_form(queue)
                    t = time.perf_counter()
                    b.run(autotune=tune, f32=True)
                    ms.append(time.perf_counter() - t)
                    assert b.form()[0] == queue
                    for s, r in zip(series, solo):
                        assert_same(results(s), r)
                took[tune] = min(ms)
        assert took[True] > 2.5 * took[False], took
    finally:
        for s in series:
            s.close()


@pytest.mark.parametrize("queue", [True, False])
def test_sorts_of_a_members_events_leave_a_captured_batch_its_buffers(queue):
    """Members transposed in tiles of 16 items per lane; the ordered side
    statistics and the two-time lists sort their events in tiles of 8, between
    the capture and the replays of the batch's graph."""
    flat = golden_member("sparse_flat")[1]
    plain = [open_member(*synth_member(i, *m)) for i, m in enumerate(MIX[:3])]
    members = plain + [flat]
    try:
        for s in members:
            s.set_tuning(80, 0, 16)
        solo = [alone(s, xg.MODE_REFERENCE) for s in members]
        with xg.Batch(members) as b:
            b.set_form(queue)
            for k in range(4):
                b.run(xg.MODE_REFERENCE, f64=True, f32=True)
                for s, r in zip(members, solo):
                    assert_same(results(s), r)
                if k >= 1:  # the graph exists
                    for s in members:
                        s.side_stats(max(s.frames // 10, 1))
                    plain[0].twotime([1, 2], static_map=True)
                    plain[2].twotime([1], mode=xg.MODE_EXACT, fetch=False)
    finally:
        for s in members:
            s.close()


def test_a_capacity_set_after_autotuning_holds_for_few_pixels():
    """48 x 48 pixels, 4,000 frames, rows of up to 100 events: a warp a row by
    default, a thread a row once the caller chose a capacity, before or after
    an autotune.  One thread a row takes several times as long here."""
    acq, dq, sq, frames = synth_member(2, 48, 4000, 0.02, 8, (10, 900))

    def int_ms(s):
        ms = []
        for _ in range(8):
            s.multitau()
            s.synchronize()
            ms.append(s.stage_times()["multitau_int_ms"])
        return min(ms)

    s = open_member(acq, dq, sq, frames)
    try:
        warp = int_ms(s)
        s.set_tuning(112, 0, 0)
        thread = int_ms(s)
        assert thread > 1.5 * warp  # or the rest says nothing
        s.autotune()
        assert int_ms(s) < 1.3 * warp  # the faster of both forms
        s.set_tuning(112, 0, 0)
        assert int_ms(s) > 1.3 * warp
    finally:
        s.close()
