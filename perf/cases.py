"""The work that a user of this correlator has it do, as measurable cases.

A case is one pass over one acquisition (or a batch of them) through the
Python front end: the frames are handed over, the correlation runs and its
results come back to the caller.  Inputs are the seeded synthetic speckle
acquisitions of `xpcs_synth` with the sizes and settings of the benchmark
configurations, the tests and the batch mix:

  sparse    photon-counting frames -> multi-tau -> g2 / stderr
  dense     CCD frames with darks and flatfield -> the same
  rows      pixel-major rows already in device memory, device results, no
            allocation
  twotime   two-time matrices per q bin, EXACT or REFERENCE order
  batch     several uneven series as one graph
"""
from __future__ import annotations

import math
import sys
from pathlib import Path

import numpy as np
import torch

_PKG = str(Path(__file__).resolve().parent.parent / "xpcs-eigen_gb300")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import xpcs_gpu as xg  # noqa: E402
import xpcs_synth as xs  # noqa: E402


def _sparse(**kw):
    case = dict(kind="sparse", n_dynamic=9, tau_min=5.0, tau_max=500.0, dpl=8, mean=0.01,
                flat=False, stride=1, average=1, source="device", push=0, block=0, f32=False,
                side=False, g2ipif=False)
    case.update(kw)
    return case


def listed():
    return [
        # a look at the first frames of a small region while the sample is being aligned: all
        # latency, every result wanted, the per-pixel arrays too
        _sparse(name="preview_64", width=64, height=64, frames=200, n_dynamic=4, mean=0.05, dpl=4,
                tau_min=2.0, tau_max=50.0, source="host", g2ipif=True),
        # an ordinary short acquisition (the 512 x 512 benchmark configuration)
        _sparse(name="series_512", width=512, height=512, frames=1000, mean=0.01, dpl=4,
                tau_min=20.0, tau_max=20.0),
        # the headline: a 1 Mpx detector, 10,000 frames, rows of about 50 events
        _sparse(name="series_1mpx", width=1024, height=1024, frames=10000, n_dynamic=18,
                mean=0.005),
        # few pixels, many photons each: rows of about 740 events, an odd detector region
        _sparse(name="long_rows", width=263, height=251, frames=16000, n_dynamic=12, mean=0.0465,
                tau_min=2.0, tau_max=2000.0),
        # flatfield and frame averaging: values are no integers, every float sum in order
        _sparse(name="flat_average", width=509, height=387, frames=1500, mean=0.02, flat=True,
                average=2),
        # frames pushed as they arrive from pinned memory, transposed block by block
        _sparse(name="stream_512", width=512, height=512, frames=5000, mean=0.01, source="pinned",
                push=64, block=512),
        # what the corr driver computes for its analysis file: float32 results in the
        # reference's order beside the float64 ones, and the filter's side statistics
        _sparse(name="corr_outputs", width=640, height=480, frames=2000, n_dynamic=12, mean=0.02,
                source="host", f32=True, side=True),
        # a CCD: darks, threshold, gain; every kept value a float
        dict(name="dense_ccd", kind="dense", width=960, height=960, frames=2000, n_dynamic=18,
             mean=0.02, dpl=8, tau_min=5.0, tau_max=500.0, darks=100, flat=True, average=1),
        # rows another program holds on the device (an acquisition loop that must not allocate)
        dict(name="rows_device", kind="rows", width=256, height=250, frames=3000, n_dynamic=9,
             mean=0.015, dpl=8, tau_min=5.0, tau_max=500.0, flat=False),
        # two-time, integer Gram on the tensor cores
        dict(name="twotime_exact", kind="twotime", width=512, height=512, frames=1536,
             n_dynamic=9, mean=0.01, tau_min=2.0, tau_max=2000.0, exact_mode=True,
             static_map=False, average=False, window=8),
        # two-time in the reference's float32 order, static-map smoothing
        dict(name="twotime_reference", kind="twotime", width=256, height=256, frames=701,
             n_dynamic=6, mean=0.02, tau_min=2.0, tau_max=500.0, exact_mode=False,
             static_map=True, average=False, window=8),
        # the uneven mix of a scan: 12 series of different sizes, new frames every time
        dict(name="batch_12", kind="batch", members=12, side_min=192, side_max=640,
             frames_min=500, frames_max=6000, mean_min=0.002, mean_max=0.04),
    ]


def _logint(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["sparse", "sparse", "sparse", "flat", "stream", "corr", "dense", "rows",
                       "exact", "reference", "batch"])
    w, h = _logint(rng, 48, 1024), _logint(rng, 48, 1024)
    tau = dict(tau_min=2.0, tau_max=float(_logint(rng, 20, 2000)))
    nq = rng.randint(3, 18)
    dpl = rng.choice([4, 8])
    if kind in ("sparse", "flat", "stream", "corr"):
        frames = _logint(rng, 200, 16000)
        mean = math.exp(rng.uniform(math.log(0.002), math.log(0.05)))
        most = {"sparse": 4e7, "flat": 8e6, "stream": 1.2e7, "corr": 1.2e7}[kind]  # events
        mean = max(min(mean, most / (w * h * frames)), 2e-4)
        frames = max(200, min(frames, int(most / (w * h * mean))))
        extra = {"sparse": dict(source=rng.choice(["device", "host"])),
                 "flat": dict(flat=rng.random() < 0.7, average=rng.choice([1, 2, 3]),
                              stride=rng.choice([1, 2])),
                 "stream": dict(source="pinned", push=rng.choice([1, 16, 64, 100]),
                                block=rng.choice([256, 512])),
                 "corr": dict(source="host", f32=True, side=True)}[kind]
        if kind == "flat":
            frames = max(100, frames // (extra["average"] * extra["stride"]))
        if kind == "stream":
            frames = min(frames, 300 * extra["push"])
        return _sparse(width=w, height=h, frames=frames, mean=mean, n_dynamic=nq, dpl=dpl,
                       g2ipif=w * h < 20000, **tau, **extra)
    if kind == "dense":
        frames = max(100, min(_logint(rng, 100, 4000), int(1.5e9 / (w * h))))
        return dict(kind="dense", width=w, height=h, frames=frames, n_dynamic=nq, mean=0.02,
                    dpl=dpl, darks=rng.choice([10, 50, 100]), flat=rng.random() < 0.8,
                    average=rng.choice([1, 1, 1, 2]), **tau)
    if kind == "rows":
        w, h = min(w, 400), min(h, 400)
        frames = _logint(rng, 200, 6000)
        mean = min(math.exp(rng.uniform(math.log(0.002), math.log(0.05))),
                   2.8e6 / (w * h * frames))
        return dict(kind="rows", width=w, height=h, frames=frames, n_dynamic=nq, mean=mean,
                    dpl=dpl, flat=rng.random() < 0.5, **tau)
    if kind == "exact":
        return dict(kind="twotime", width=min(w, 512), height=min(h, 512),
                    frames=_logint(rng, 100, 1500), n_dynamic=min(nq, 9),
                    mean=rng.choice([0.003, 0.01, 0.03]), exact_mode=True,
                    static_map=rng.random() < 0.3, average=rng.random() < 0.3,
                    window=rng.choice([1, 4, 8]), **tau)
    if kind == "reference":
        return dict(kind="twotime", width=min(w, 256), height=min(h, 256),
                    frames=_logint(rng, 60, 700), n_dynamic=min(nq, 6),
                    mean=rng.choice([0.005, 0.02, 0.05]), exact_mode=False,
                    static_map=rng.random() < 0.5, average=rng.random() < 0.5,
                    window=rng.choice([1, 4, 8]), **tau)
    return dict(kind="batch", members=rng.randint(3, 12), side_min=rng.choice([64, 128, 192]),
                side_max=rng.randint(256, 600), frames_min=rng.randint(200, 600),
                frames_max=rng.randint(1000, 5000), mean_min=0.002, mean_max=0.03)


# ------------------------------------------------------------------ inputs


def _acq(c, seed, frames=None, **kw):
    return xs.Acquisition(width=c["width"], height=c["height"], frames=frames or c["frames"],
                          n_static=2 * c["n_dynamic"], n_dynamic=c["n_dynamic"], mean=c["mean"],
                          tau_min=c["tau_min"], tau_max=c["tau_max"], seed=1 + int(seed),
                          dpl=c.get("dpl", 4), **kw)


def _gain(c):
    return dict(gain_min=0.9, gain_max=1.1) if c.get("flat") else {}


def _sparse_acq(c, seed):
    return _acq(c, seed, c["frames"] * c["stride"] * c["average"], **_gain(c))


def _dense_acq(c, seed):
    return _acq(c, seed, c["frames"] * c["average"], dense=True, dark_frames=c["darks"], **_gain(c))


def _batch_acqs(c, seed):
    rng = np.random.default_rng(int(seed) + 17)

    def between(lo, hi):
        return float(np.exp(rng.uniform(np.log(c[lo]), np.log(c[hi]))))

    # the sizes are the case's, not the seed's: they come from a generator of their own
    sizes = np.random.default_rng(c["members"])
    acqs = []
    for _ in range(c["members"]):
        rng, keep = sizes, rng
        side, frames = int(between("side_min", "side_max")), int(between("frames_min", "frames_max"))
        mean, q = between("mean_min", "mean_max"), int(rng.integers(4, 19))
        dpl = int(rng.choice([4, 8]))
        rng = keep
        acqs.append(xs.Acquisition(width=side, height=side, frames=frames, n_static=2 * q,
                                   n_dynamic=q, mean=mean, tau_min=2.0, tau_max=2000.0, dpl=dpl,
                                   seed=int(rng.integers(1, 1 << 40))))
    return acqs


def _rows_of(acq, flat):
    """Pixel-major rows of a sparse acquisition: row_ptr, frame, value on the GPU."""
    d = xs.DeviceFrames(acq)
    nnz, idx, val = (torch.from_numpy(a.astype(np.int64)).cuda() for a in d.to_host())
    d.close()
    frame = torch.repeat_interleave(torch.arange(acq.frames, device="cuda"), nnz)
    pix, order = torch.sort(idx, stable=True)
    row_ptr = torch.searchsorted(pix, torch.arange(acq.width * acq.height + 1, device="cuda"))
    value = val[order].to(torch.float32)
    if flat:
        gain = torch.from_numpy(xs.maps(acq)[2].ravel()).cuda()
        value = (value.double() * gain[pix]).float()
    return row_ptr, frame[order].to(torch.int32), value


def prepare(case, seed):
    c = case
    if c["kind"] == "sparse":
        acq = _sparse_acq(c, seed)
        dq, sq, flat, _ = xs.maps(acq)
        s = xg.Series(c["width"], c["height"], c["frames"], c["dpl"], dq, sq,
                      flatfield=flat if c["flat"] else None, stride=c["stride"],
                      average=c["average"])
        if c["block"]:
            s.set_block_frames(c["block"])
        d = xs.DeviceFrames(acq)
        st = dict(case=c, series=s, nnz=d.nnz, frames=d)
        if c["source"] != "device":
            _, idx, val = d.to_host()
            d.close()
            if c["source"] == "pinned":
                st["pinned"] = (torch.from_numpy(idx).pin_memory(), torch.from_numpy(val).pin_memory())
                idx, val = (t.numpy() for t in st["pinned"])
            st.update(idx=idx, val=val, off=np.concatenate([[0], np.cumsum(d.nnz, dtype=np.int64)]))
        return st
    if c["kind"] == "dense":
        acq = _dense_acq(c, seed)
        dq, sq, flat, _ = xs.maps(acq)
        d = xs.DeviceDenseFrames(acq)
        s = xg.Series(c["width"], c["height"], c["frames"], c["dpl"], dq, sq,
                      flatfield=flat if c["flat"] else None, average=c["average"], dense=True,
                      lld=0.0, sigma=3.0)
        s.set_dark(d.to_host(0, c["darks"]))
        return dict(case=c, series=s, frames=d)
    if c["kind"] == "rows":
        acq = _acq(c, seed, **_gain(c))
        row_ptr, frame, value = _rows_of(acq, c["flat"])
        D, P = xg.delay_schedule(c["frames"], c["dpl"])[0].size, c["width"] * c["height"]
        out = [torch.empty((D, P), dtype=torch.float32, device="cuda") for _ in range(3)]
        return dict(case=c, row_ptr=row_ptr, frame=frame, value=value, out=out)
    if c["kind"] == "twotime":
        acq = _acq(c, seed)
        dq, sq, _, _ = xs.maps(acq)
        s = xg.Series(c["width"], c["height"], c["frames"], 4, dq, sq)
        return dict(case=c, series=s, frames=xs.DeviceFrames(acq),
                    qbins=list(range(1, c["n_dynamic"] + 1)))
    members = []
    for acq in _batch_acqs(c, seed):
        dq, sq, _, _ = xs.maps(acq)
        members.append((xg.Series(acq.width, acq.height, acq.frames, acq.dpl, dq, sq),
                        xs.DeviceFrames(acq)))
    return dict(case=c, members=members, batch=xg.Batch([s for s, _ in members]))


def run(state):
    c = state["case"]
    if c["kind"] == "rows":
        r, f, v = state["row_ptr"], state["frame"], state["value"]
        out = state["out"]
        xg.multitau2_noalloc(r.data_ptr(), f.data_ptr(), v.data_ptr(), r.numel() - 1, f.numel(),
                             c["frames"], c["dpl"], xg.MODE_REFERENCE,
                             *[t.data_ptr() for t in out],
                             stream=torch.cuda.current_stream().cuda_stream)
        return out
    if c["kind"] == "batch":
        for s, d in state["members"]:
            s.reset()
            s.ingest_sparse_device(d.nnz, d.idx, d.val)
        state["batch"].run(f64=True)
        return [s.normalized()[:2] for s, _ in state["members"]]
    s = state["series"]
    s.reset()
    if c["kind"] == "dense":
        d = state["frames"]
        s.ingest_dense_device(d.frame_ptr(c["darks"]), c["frames"] * c["average"])
    elif c.get("source", "device") == "device":
        d = state["frames"]
        s.ingest_sparse_device(d.nnz, d.idx, d.val)
    else:
        nnz, idx, val, off = state["nnz"], state["idx"], state["val"], state["off"]
        step = c["push"] or nnz.size
        for k in range(0, nnz.size, step):
            e = min(k + step, nnz.size)
            s.ingest_sparse(nnz[k:e], idx[off[k]:off[e]], val[off[k]:off[e]])
    if c["kind"] == "twotime":
        r = s.twotime(state["qbins"], static_map=c["static_map"], average=c["average"],
                      window=c["window"], mode=xg.MODE_EXACT if c["exact_mode"]
                      else xg.MODE_REFERENCE)
        return [r["sg"], r["g2full"], r["g2partials"], [r["c2t"][q] for q in sorted(r["c2t"])]]
    s.multitau()
    f32 = c.get("f32", False)
    out = {"norm": list(s.normalize(f64=True, f32=f32)[:4 if f32 else 2])}
    if c.get("side"):
        out["side"] = list(s.side_stats(max(c["frames"] // 10, 1)))
    if c.get("g2ipif"):
        out["g2ipif"] = list(s.g2ipif())
    return out


# -------------------------------------------------------------------- work


def _schedule(frames, dpl):
    """[(level, [delays in frames])]: 2 dpl delays of step 1, then dpl of each step 2^k."""
    last = 0
    if frames >= 2 * dpl:
        last = int(math.floor(math.log2(frames) - math.log2(1.0 + 1.0 / dpl)) - math.log2(dpl))
    t, levels = 0, []
    for lv in range(last + 1):
        taus = []
        for _ in range(2 * dpl if lv == 0 else dpl):
            if t + 2 * (1 << lv) > frames:
                break
            t += 1 << lv
            taus.append(t)
        if taus:
            levels.append((lv, taus))
    return levels


def _multitau_work(P, frames, dpl, mean, events):
    """Adds of the row merges, products and adds of the pairs that exist, quotients."""
    flops, D = 2.0 * events, 0
    for lv, taus in _schedule(frames, dpl):
        entries = P * (frames >> lv) * (1.0 - math.exp(-mean * (1 << lv)))
        flops += entries * (1 + 2 * len(taus) * (1.0 - math.exp(-mean * (1 << lv))))
        D += len(taus)
    return flops + 3.0 * D * P, D


def work(case):
    c = case
    if c["kind"] == "batch":
        parts = [work(_sparse(width=a.width, height=a.height, frames=a.frames, mean=a.mean,
                              n_dynamic=a.n_dynamic, dpl=a.dpl)) for a in _batch_acqs(c, 0)]
        return {k: sum(p[k] for p in parts) for k in ("bytes", "flops")}
    P, F, nq = c["width"] * c["height"], c["frames"], c["n_dynamic"]
    raw = F * c.get("average", 1) if c["kind"] != "twotime" else F
    events = P * raw * c["mean"] / (1.0 + c["mean"])
    if c["kind"] == "twotime":
        rows = 0.95 * P
        return {"bytes": 6.0 * events + 4.0 * nq * F * F,
                "flops": rows * F * (F + 1) if c["exact_mode"] else 2.0 * events * F * c["mean"]}
    flops, D = _multitau_work(P, F, c["dpl"], c["mean"], events)
    if c["kind"] == "rows":
        return {"bytes": 8.0 * events + 8.0 * P + 12.0 * D * P, "flops": flops}
    out = 16.0 * D * nq * (1.5 if c.get("f32") else 1.0)
    if c.get("g2ipif"):
        out += 12.0 * D * P
    if c.get("side"):
        out += 4.0 * P + 8.0 * F + 4.0 * 11 * 2 * nq
    read = 2.0 * P * raw if c["kind"] == "dense" else 6.0 * events
    return {"bytes": read + out, "flops": flops + 12.0 * D * P}


# ------------------------------------------------- the results in 64 bits


def _merge(pix, frame, value):
    """Events of one pixel and frame summed; sorted by (pixel, frame)."""
    span = int(frame.max()) + 1 if frame.numel() else 1
    key, inv = torch.unique(pix * span + frame, return_inverse=True)
    return key // span, key % span, torch.zeros(key.numel(), dtype=torch.float64,
                                                device="cuda").index_add_(0, inv, value)


def _multitau64(P, F, dpl, pix, frame, value):
    """G2, IP, IF [D][P] of rows sorted by (pixel, frame), REFERENCE semantics: the partner of
    an event is looked up by halving over the row's whole buffer, stale entries included."""
    n0 = torch.bincount(pix, minlength=P)
    start = torch.cumsum(n0, 0) - n0
    buf = frame.clone()
    steps = int(n0.max()).bit_length() + 1 if pix.numel() else 0
    out = ([], [], [])
    lf, at = F, 0
    for lv, taus in _schedule(F, dpl):
        if lv != at:
            lf, at = lf // 2, lv
            frame = frame >> 1
            pix, frame, value = (t[frame < lf] for t in (pix, frame, value))
            pix, frame, value = _merge(pix, frame, 0.5 * value)
        n = torch.bincount(pix, minlength=P)
        rank = torch.arange(pix.numel(), device="cuda") - (torch.cumsum(n, 0) - n)[pix]
        if pix.numel():
            buf[start[pix] + rank] = frame
        first, left = torch.zeros_like(frame), n0[pix]
        for _ in range(steps):
            half = left >> 1
            mid = (start[pix] + first + half).clamp(max=max(buf.numel() - 1, 0))
            right = (left > 0) & (buf[mid] < frame)
            first = torch.where(right, first + half + 1, first)
            left = torch.where(right, left - half - 1, torch.where(left > 0, half, left))
        found = first == rank
        key = pix * (lf + 1) + frame
        for t in taus:
            tau, den = t >> lv, float(max(lf - (t >> lv), 1))
            early, late = frame < lf - tau, frame >= tau
            j = torch.searchsorted(key, key + tau).clamp(max=max(key.numel() - 1, 0))
            pair = early & (key[j] == key + tau) & found[j] if key.numel() else early
            for o, sel, v in ((out[0], pair, value * value[j] if key.numel() else value),
                              (out[1], early, value), (out[2], late, value)):
                o.append(torch.zeros(P, dtype=torch.float64, device="cuda").index_add_(
                    0, pix[sel], v[sel]) / den)
    return [torch.stack(o) for o in out]


def _norm64(dq, sq, G2, IP, IF):
    dq, sq = (torch.from_numpy(np.ascontiguousarray(a.ravel()).astype(np.int64)).cuda()
              for a in (dq, sq))
    valid = ((dq > 0) & (sq > 0)).nonzero().ravel()
    q_ids = torch.unique(dq[valid]).tolist()
    g2, se = (torch.zeros((G2.shape[0], len(q_ids)), dtype=torch.float64, device="cuda")
              for _ in range(2))
    for q in q_ids:
        pix = valid[dq[valid] == q]
        ratios = []
        for sb in torch.unique(sq[pix]).tolist():
            p = pix[sq[pix] == sb]
            ratios.append(G2[:, p].mean(1) / (IP[:, p].mean(1) * IF[:, p].mean(1)))
        g2[:, q - 1] = torch.nanmean(torch.stack(ratios), 0)
        x = torch.nan_to_num(G2[:, pix] / (IP[:, pix] * IF[:, pix]), nan=0.0)
        m2 = ((x - x.mean(1, keepdim=True)) ** 2).sum(1)
        se[:, q - 1] = (m2 / pix.numel()).sqrt() / math.sqrt(pix.numel())
    return g2, se


def _side64(c, dq, sq, pix, frame, value):
    P, F, win = c["width"] * c["height"], c["frames"], max(c["frames"] // 10, 1)
    sb = torch.from_numpy(np.where(dq > 0, sq, 0).ravel().astype(np.int64)).cuda()
    S = int(sb.max())

    def add(n, at, v):
        return torch.zeros(n, dtype=torch.float64, device="cuda").index_add_(0, at, v)

    ppb = torch.bincount(sb, minlength=S + 1)[1:].double()
    bins = sb[pix] - 1
    w = frame // win
    keep = w < F // win
    part = add((F // win) * S, w[keep] * S + bins[keep], value[keep]).reshape(F // win, S)
    fs = torch.stack([torch.arange(1, F + 1, device="cuda").double(), add(F, frame, value) / P])
    return [add(P, pix, value).reshape(c["height"], c["width"]) / F, fs,
            (add(S, bins, value) / (ppb * F)).reshape(1, S), part / (ppb * win)]


def _sparse_events(c, acq, dq, sq, flat):
    """Filtered, merged events (pixel, filter frame, value) of a sparse series."""
    d = xs.DeviceFrames(acq)
    nnz, idx, val = (torch.from_numpy(a.astype(np.int64)).cuda() for a in d.to_host())
    d.close()
    r = torch.repeat_interleave(torch.arange(acq.frames, device="cuda"), nnz)
    stride, average = c.get("stride", 1), c.get("average", 1) if c["kind"] == "sparse" else 1
    group = stride * average
    live = torch.from_numpy(((dq > 0) & (sq > 0)).ravel()).cuda()
    keep = live[idx] & (r % group % stride == 0)
    pix, frame, value = idx[keep], (r // group)[keep], val[keep].double()
    if c.get("flat"):
        value = value * torch.from_numpy(flat.ravel()).cuda()[pix]
    return _merge(pix, frame, value / average)


def _dense_events(c, acq, dq, sq, flat):
    d = xs.DeviceDenseFrames(acq)
    P, n = d.P, c["darks"]
    gain = torch.from_numpy(flat.ravel()).cuda() if c["flat"] else torch.ones(
        P, dtype=torch.float64, device="cuda")
    live = torch.from_numpy(((dq > 0) & (sq > 0)).ravel()).cuda()
    avg, m2 = (torch.zeros(P, dtype=torch.float64, device="cuda") for _ in range(2))
    for i, raw in enumerate(d.to_host(0, n)):
        x = torch.from_numpy(raw).cuda().double() * gain
        old = avg
        avg = old + (x - old) / (i + 1)
        m2 = m2 + (x - old) * (x - avg)
    # which values are kept is decided in float32, as the threshold is defined
    thresh = (3.0 * (m2 / n).sqrt()).float()
    got = [], [], []
    for f0 in range(0, acq.frames, 256):
        raw = torch.from_numpy(d.to_host(n + f0, min(256, acq.frames - f0))).cuda().double() - avg
        f, p = ((raw.float() > thresh) & live).nonzero(as_tuple=True)
        for g, x in zip(got, (p, (f + f0) // c["average"], raw[f, p] * gain[p] / c["average"])):
            g.append(x)
    d.close()
    return _merge(*[torch.cat(g) for g in got])


def _series64(c, acq, dense=False):
    dq, sq, flat, _ = xs.maps(acq)
    ev = (_dense_events if dense else _sparse_events)(c, acq, dq, sq, flat)
    three = _multitau64(c["width"] * c["height"], c["frames"], c["dpl"], *ev)
    out = {"norm": list(_norm64(dq, sq, *three)) * (2 if c.get("f32") else 1)}
    if c.get("side"):
        out["side"] = _side64(c, dq, sq, *ev)
    if c.get("g2ipif"):
        out["g2ipif"] = three
    return out


def _twotime64(c, acq):
    dq, sq, _, _ = xs.maps(acq)
    F = c["frames"]
    pix, frame, value = _sparse_events(c, acq, dq, sq, None)
    V = torch.zeros((acq.width * acq.height, F), dtype=torch.float64, device="cuda")
    V[pix, frame] = value
    q_of, s_of = (torch.from_numpy(np.where((dq > 0) & (sq > 0), a, 0).ravel().astype(np.int64)
                                   ).cuda() for a in (dq, sq))
    sgs, full, part, mats = [], [], [], []
    tp, win = max(0, (F - c["window"]) // c["window"]), c["window"]
    for q in range(1, c["n_dynamic"] + 1):
        here = (q_of == q).nonzero().ravel()
        groups = ([here[s_of[here] == b] for b in torch.unique(s_of[here]).tolist()]
                  if c["static_map"] else [here])
        rows = []
        for g in groups:
            sg = V[g].mean(0)
            sg = sg.mean(0, keepdim=True) if c["average"] else sg
            sgs.append(sg)
            rows.append(V[g] / torch.where(sg > 0, sg, torch.ones_like(sg)))
        X = torch.cat(rows)
        C = torch.triu(X.T @ X) / here.numel()
        mats.append(C.cpu())
        diag = [torch.diagonal(C, k) for k in range(F)]
        full.append(torch.stack([x.mean() for x in diag]))
        part.append(torch.stack([torch.cat([diag[k], diag[k].new_zeros(k)])[:tp * win].reshape(
            tp, win).sum(1) / win for k in range(win)]))
    return [torch.stack(sgs), torch.stack(full, 1), torch.stack(part, 2), mats]


def exact(case, seed):
    c = case
    if c["kind"] == "sparse":
        return _series64(c, _sparse_acq(c, seed))
    if c["kind"] == "dense":
        return _series64(c, _dense_acq(c, seed), dense=True)
    if c["kind"] == "twotime":
        return _twotime64(c, _acq(c, seed))
    if c["kind"] == "rows":
        row_ptr, frame, value = _rows_of(_acq(c, seed, **_gain(c)), c["flat"])
        P = c["width"] * c["height"]
        pix = torch.repeat_interleave(torch.arange(P, device="cuda"), row_ptr[1:] - row_ptr[:-1])
        return _multitau64(P, c["frames"], c["dpl"], pix, frame.long(), value.double())
    return [_series64(dict(kind="sparse", width=a.width, height=a.height, frames=a.frames,
                           dpl=a.dpl), a)["norm"] for a in _batch_acqs(c, seed)]
