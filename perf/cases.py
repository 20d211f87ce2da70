"""Performance cases of the CRV engine: the calls its users make, from the smallest to the largest, on synthetic inputs
of the workload's distributions.

  chain    ResidentChain.run, one batch of steps -> coincidence clusters through the captured graph: FP32-mixed on the
           one-module detector (the main line), FP64-plain, the full 86-module detector, the lookup-table photon model
  fit      GraphFitter.fit, the batched pulse fit of uneven waveforms, FP32-mixed and FP64
  substeps SubstepEngine.run, the lookup-table photon model's rows -> photons, FP64 and FP32-mixed
  dropin   chain.charges -> digis -> reco_waveforms -> clusters on host tables, the reference's own call sequence
  synth    waveform.synthesize on host charges with the caller's TDC0 and no noise (FP64)

Outputs that come from keyed random draws (chain, substeps, dropin) or from a fit that stops on a schedule (fit) have
no value that plain 64-bit arithmetic gives; synth has, and exact() gives it.
"""
import math
import os
import sys

import numpy as np
import torch

_PKG = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "mu2e-fastsim_gb300")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

from crvgpu import chain as CH  # noqa: E402
from crvgpu import config as CF  # noqa: E402
from crvgpu import geometry as GM  # noqa: E402
from crvgpu import lookup as LK  # noqa: E402
from crvgpu import waveform as WF  # noqa: E402
from crvgpu.params import make_params  # noqa: E402
from crvgpu.pulsefit import GraphFitter  # noqa: E402
from crvgpu.resident import ChainCaps, ResidentChain  # noqa: E402
from crvgpu.response import DeviceSteps, upload_steps  # noqa: E402

DEV = "cuda"
FULL_MODULES = 86          # the full detector of the benchmark's full-scale leg
# stage counts per step of the workload (measured): photons, charges, digi slots, digis, pulses
PER_STEP = {"module": (255, 101, 3.9, 3.5, 3.6), "full": (260, 103, 3.9, 3.5, 3.6), "lookup": (313, 123, 6.2, 3.5, 3.6)}


def listed():
    return [
        # one trigger's worth of events: every launch of the chain, hardly any work in it (express jobs of the server)
        {"name": "chain_16", "kind": "chain", "events": 16, "precision": "fp32", "detector": "module",
         "pixel_id": "truncate"},
        # a serving slot's chunk (crvgpu.serve's default)
        {"name": "chain_2048", "kind": "chain", "events": 2048, "precision": "fp32", "detector": "module",
         "pixel_id": "truncate"},
        # the benchmark's default batch
        {"name": "chain_65536", "kind": "chain", "events": 65536, "precision": "fp32", "detector": "module",
         "pixel_id": "truncate"},
        # the bit-exact FP64 chain, an uneven batch, with the reference's default pixel rule
        {"name": "chain_fp64_1500", "kind": "chain", "events": 1500, "precision": "fp64", "detector": "module",
         "pixel_id": "lrint"},
        # the full detector: 5,504 counters, about 2,800 steps per event
        {"name": "full_512", "kind": "chain", "events": 512, "precision": "fp32", "detector": "full",
         "pixel_id": "truncate"},
        # the production photon model (lookup tables) inside the resident chain
        {"name": "lookup_chain_2048", "kind": "chain", "events": 2048, "precision": "fp32", "detector": "lookup",
         "pixel_id": "truncate"},
        # the batched pulse fit of uneven waveforms (the workload's batching configuration), mixed and plain
        {"name": "fit_fp32_262144", "kind": "fit", "waveforms": 262144, "precision": "fp32"},
        {"name": "fit_fp64_10007", "kind": "fit", "waveforms": 10007, "precision": "fp64"},
        # lookup-table photons of muon crossings, mixed and plain
        {"name": "substeps_fp32_200000", "kind": "substeps", "rows": 200000, "precision": "fp32", "decay": 0.0},
        {"name": "substeps_fp64_20011", "kind": "substeps", "rows": 20011, "precision": "fp64", "decay": 7.4},
        # the reference's own calls on host tables
        {"name": "dropin_1000", "kind": "dropin", "events": 1000, "precision": "fp32"},
        # waveform synthesis on host charges
        {"name": "synth_30000", "kind": "synth", "channels": 30000},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    k = rng.choices(("module32", "module64", "full", "lookup", "fit32", "fit64", "sub32", "sub64", "dropin", "synth"),
                    (30, 12, 8, 10, 10, 7, 6, 6, 6, 5))[0]
    pix = rng.choice(("truncate", "lrint"))
    if k == "module32":
        return {"kind": "chain", "events": _log(rng, 8, 65536), "precision": "fp32", "detector": "module",
                "pixel_id": pix}
    if k == "module64":
        return {"kind": "chain", "events": _log(rng, 8, 4096), "precision": "fp64", "detector": "module",
                "pixel_id": pix}
    if k == "full":
        return {"kind": "chain", "events": _log(rng, 2, 640), "precision": "fp32", "detector": "full",
                "pixel_id": pix}
    if k == "lookup":
        return {"kind": "chain", "events": _log(rng, 8, 4096), "precision": "fp32", "detector": "lookup",
                "pixel_id": pix}
    if k in ("fit32", "fit64"):
        return {"kind": "fit", "waveforms": _log(rng, 100, 400000 if k == "fit32" else 30000),
                "precision": "fp" + k[3:]}
    if k in ("sub32", "sub64"):
        return {"kind": "substeps", "rows": _log(rng, 200, 400000 if k == "sub32" else 60000),
                "precision": "fp" + k[3:], "decay": rng.choice((0.0, 7.4))}
    if k == "dropin":
        return {"kind": "dropin", "events": _log(rng, 8, 4000), "precision": rng.choice(("fp32", "fp64"))}
    return {"kind": "synth", "channels": _log(rng, 100, 60000)}


# ---- inputs -----------------------------------------------------------------------------------------------------

def _device_steps(case, seed, geom):
    """Steps of the workload (crvgpu.geometry.synthetic_steps' distributions), generated on the device."""
    g = torch.Generator(device=DEV)
    g.manual_seed(seed)
    e, nb = case["events"], geom.nbars
    mean = _mean_steps(case["detector"])
    per = torch.poisson(torch.full((e,), mean, device=DEV, dtype=torch.float64), generator=g).to(torch.int64)
    n = int(per.sum())
    first = torch.cumsum(per, 0) - per
    bar = torch.randint(0, nb, (n,), generator=g, device=DEV)
    ax = torch.from_numpy(np.asarray(geom.local_to_world, np.int64)).to(DEV)[bar]
    half = torch.from_numpy(np.asarray(geom.halflen, float)).to(DEV)[bar]
    pos = torch.from_numpy(np.asarray(geom.center, float)).to(DEV)[bar].clone()
    u = 2.0 * torch.rand((n, 3), generator=g, device=DEV, dtype=torch.float64) - 1.0
    for k in range(3):
        a = ax[:, k:k + 1]
        pos.scatter_add_(1, a, u[:, k:k + 1] * half.gather(1, a))
    ln = 5.0 + 20.0 * torch.rand(n, generator=g, device=DEV, dtype=torch.float64)
    z = torch.randn(n, generator=g, device=DEV, dtype=torch.float64)
    edep = (3.6 - 0.3 * torch.log(z * z)) * ln / 19.8
    t = 1700.0 * torch.rand(n, generator=g, device=DEV, dtype=torch.float64)
    one = torch.ones(e, dtype=torch.int32, device=DEV)
    f32 = lambda a: a.to(torch.float32).contiguous()  # noqa: E731
    return DeviceSteps(x=f32(pos[:, 0]), y=f32(pos[:, 1]), z=f32(pos[:, 2]), t=f32(t), edep=f32(edep),
                       bar=bar.to(torch.int32), ev_event=torch.arange(e, dtype=torch.int32, device=DEV), ev_subrun=one,
                       ev_run=one.clone(), ev_first=first, ev_nsteps=per.to(torch.int32), nsteps=n, nevents=e,
                       max_steps=int(per.max()))


def _mean_steps(detector):
    return 60.0 + 32.0 * FULL_MODULES if detector == "full" else 40.0


def _caps(events, detector):
    """Capacities from the configuration alone, as a program sets them before it has seen a batch."""
    mean = _mean_steps(detector)
    steps = int(mean * events + 8.0 * math.sqrt(mean * events)) + 64
    ph, ch, sl, dg, pu = (int(1.2 * v * steps) + 40000 for v in PER_STEP[detector])
    return ChainCaps(events=events, steps=steps, photons=ph, charges=ch, slots=sl, digis=dg, pulses=pu,
                     max_steps_per_event=int(mean + 8.0 * math.sqrt(mean)))


def _rows(buffers, n):
    """The first n rows of every device buffer, cleared."""
    out = {k: v[:n] for k, v in buffers.items()}
    for v in out.values():
        v.zero_()
    return out


def _prepare_chain(case, seed):
    lookup = extra = None
    if case["detector"] == "lookup":
        geom, cond, tables, lcfg, steps, pdg = LK.synthetic_module_lookup(case["events"], seed=seed)
        ds = upload_steps(steps, nbars=geom.nbars)
        cfg = CF.ChainConfig(precision=case["precision"], lookup=lcfg, sipm=CF.SiPMConfig(pixel_id=case["pixel_id"]))
        lookup = LK.LookupModel(geom, lcfg, tables, cond.deviation, precision=case["precision"])
        extra = lookup.upload_steps(steps, pdg)
    else:
        geom = GM.module_geometry(FULL_MODULES if case["detector"] == "full" else 1)
        cond = GM.default_conditions(geom)
        ds = _device_steps(case, seed, geom)
        cfg = CF.ChainConfig(precision=case["precision"], sipm=CF.SiPMConfig(pixel_id=case["pixel_id"]))
    rc = ResidentChain(CH.ChainEngine(geom, cond, cfg), _caps(case["events"], case["detector"]), real_dtype=ds.x.dtype,
                       graph=True, lookup=lookup)
    # a serving program captures its graph before the first job (crvgpu.serve); the batch of this warm-up is empty
    none = DeviceSteps(*[getattr(ds, k)[:0] for k in ("x", "y", "z", "t", "edep", "bar", "ev_event", "ev_subrun",
                                                      "ev_run", "ev_first", "ev_nsteps")], nsteps=0, nevents=0,
                       max_steps=0)
    rc.run(none, 1, lookup_steps=None if extra is None else {k: v[:0] for k, v in extra.items()})
    # the chain's own cluster and member buffers, more rows of them than a batch of this size fills
    e = case["events"]
    ncl, nm = (64 + 3 * e, 512 + 40 * e) if case["detector"] == "full" else (64 + e // 4, 512 + 2 * e)
    return {"rc": rc, "ds": ds, "seed": seed & 0xFFFFFF, "extra": extra,
            "out": {"clusters": _rows(rc.cl, min(ncl, rc.caps.pulses)), "members": _rows(rc.mem, min(nm, rc.caps.pulses))}}


def _run_chain(s):
    r = s["rc"].run(s["ds"], s["seed"], lookup_steps=s["extra"])
    return {**s["out"], "counts": r.counts}


def _prepare_fit(case, seed):
    """Waveforms of 32-512 samples with 1-12 Gumbel pulses of 5-500 PE on a noisy pedestal."""
    g = torch.Generator(device=DEV)
    g.manual_seed(seed)
    n, area, period = case["waveforms"], 400.0, CF.PERIOD
    rand = lambda *sh: torch.rand(*sh, generator=g, device=DEV)  # noqa: E731
    # five length classes as the benchmark has them, with ragged lengths among them
    lens = torch.tensor([32, 64, 128, 256, 512], device=DEV)[torch.randint(0, 5, (n,), generator=g, device=DEV)]
    lens = torch.where(rand(n) < 0.3, lens - torch.randint(0, 20, (n,), generator=g, device=DEV), lens)
    off = torch.cumsum(lens, 0) - lens
    ns = int(lens.sum())
    start = torch.randint(0, 200, (n,), generator=g, device=DEV)
    wf = torch.repeat_interleave(torch.arange(n, device=DEV), lens)
    t = ((start[wf] + torch.arange(ns, device=DEV) - off[wf]) * period).float()
    y = 100.0 + 2.0 * torch.randn(ns, generator=g, device=DEV)
    npul = torch.randint(1, 13, (n,), generator=g, device=DEV)
    for k in range(12):
        u = rand(3, n)
        beta = 10.0 + 15.0 * u[1]
        amp = torch.where(npul > k, torch.exp(math.log(5.0) + u[0] * math.log(100.0)) * area / beta,
                          torch.zeros_like(beta))
        z = (t - ((start + u[2] * lens) * period).float()[wf]) / beta[wf]
        y += amp[wf] * torch.exp(-z - torch.exp(-z))
    one = torch.ones(n, dtype=torch.float64, device=DEV)
    P = make_params(reco=CF.RecoConfig(), precision=case["precision"])
    P.period = period
    gf = GraphFitter(P, n, 512 * n, 16 * n, device=DEV)
    args = (off, lens.to(torch.int32), start.to(torch.int64), 100.0 * one, area * one, area / 15.0 * one,
            torch.clamp(torch.round(y), 0, 4095).to(torch.int16))
    # the fitter's own pulse buffers (8 rows a waveform; about 5 are filled) and its count
    return {"gf": gf, "args": args, "out": {"pulses": _rows(gf.out, 8 * n), "near": gf.near, "n": gf.n_out}}


def _run_fit(s):
    s["gf"].fit(*s["args"])
    return s["out"]


def _prepare_substeps(case, seed):
    """Muon crossings of a 3200 mm bar: 20 mm tracks in 0.1 mm substeps through a table of 10 x 41 x 56 position bins
    with 150 delay bins (the benchmark's table)."""
    from types import SimpleNamespace
    rng = np.random.default_rng(seed)
    n = case["rows"]
    edges = {"x": np.linspace(0, 9.89, 11), "y": np.linspace(-25.67, 25.67, 42), "z": np.linspace(-1600, 1600, 57),
             "beta": np.linspace(0.455, 1.0, 6), "theta": np.linspace(0, np.pi, 12), "phi": np.linspace(0, np.pi, 6),
             "r": np.linspace(0, 0.616, 6)}
    nb = {k: len(v) - 1 for k, v in edges.items()}

    def table(m):
        d = rng.integers(0, 4, (m, 150), dtype=np.uint8)
        e = rng.integers(0, 40, (m, 8), dtype=np.uint8)
        return SimpleNamespace(prob=np.full(m, 0.0015, np.float32), delays=d, delay_sum=d.sum(1, dtype=np.int32),
                               emis=e, emis_sum=e.sum(1, dtype=np.int32))

    m = nb["x"] * nb["y"] * nb["z"]
    L = SimpleNamespace(name="synthetic_3200", half_thickness=9.64, half_width=25.42, half_length=1600.0,
                        fiber_separation=26.0, hole_radius_x=2.0, hole_radius_y=1.0, fiber_radius=0.7,
                        corner_radius=1.75, fiber_decay_time=case["decay"], edges=edges,
                        tables={"scint": table(m), "ckscint": table(m * nb["beta"]),
                                "ckfiber": table(nb["beta"] * nb["theta"] * nb["phi"] * nb["r"] * nb["z"])})
    a = np.c_[np.full(n, -10.0), rng.uniform(-24, 24, n), rng.uniform(-1500, 1500, n)]
    d = np.c_[np.full(n, 20.0), rng.normal(0, 2, n), rng.normal(0, 2, n)]
    dl = np.linalg.norm(d, axis=1)
    nsub = np.maximum((dl / 0.1).astype(np.int64), 1)
    t0 = rng.uniform(0, 1e5, n)
    per = lambda avg: np.maximum(np.rint(rng.normal(avg, math.sqrt(avg), n) / nsub), 0).astype(np.int64)  # noqa: E731
    ck = 266.0 * (0.999 - 0.474) / (1.0 - 0.474) * 20.0
    rows = {"s": a, "d": d, "t0": t0, "t1": t0 + 0.07, "nsub": nsub, "beta": np.full(n, 0.999),
            "theta": np.arccos(np.clip(d[:, 2] / dl, -1, 1)), "dev": np.full(n, 0.94),
            "step": np.arange(n, dtype=np.int64), "chan": (np.arange(n, dtype=np.int64) % 8192) * 4,
            "n_scint": per(28610.0 * 3.4), "n_ck_s": per(ck), "n_ck_f": per(ck)}
    eng = LK.SubstepEngine(DEV)
    eng.per_row = 200.0
    return {"eng": eng, "table": LK.DeviceLookup(L), "rows": LK.DeviceRows(rows), "seed": seed & 0xFFFFFF,
            "precision": case["precision"],
            # the photon buffers that the next stage reads
            "out": [torch.zeros(200 * n, dtype=t, device=DEV) for t in (torch.int64, torch.int64, torch.float64)]}


def _run_substeps(s):
    for o, x in zip(s["out"], s["eng"].run(s["table"], s["rows"], s["seed"], precision=s["precision"])):
        o[:len(x)].copy_(x)
    return s["out"]


def _prepare_dropin(case, seed):
    geom = GM.module_geometry()
    return {"geom": geom, "cond": GM.default_conditions(geom), "cfg": CF.ChainConfig(precision=case["precision"]),
            "steps": GM.synthetic_steps(case["events"], geom, seed=seed), "seed": seed & 0xFFFFFF,
            "events": case["events"], "out": {}}


def _keep(out, key, x, rows):
    """x in the rows of a host table that the program keeps between passes."""
    x = np.asarray(x)
    if key not in out:
        out[key] = np.zeros((rows,) + x.shape[1:], x.dtype)
    out[key][:len(x)] = x


def _run_dropin(s):
    geom, cond, cfg, seed = s["geom"], s["cond"], s["cfg"], s["seed"]
    Q = CH.charges(s["steps"], None, geom, cond, cfg, None, key=seed)
    D = CH.digis(Q, cond, cfg, None, key=seed + 1)
    W = CH.reco_waveforms(D, cond)
    cl, _ = CH.clusters(W, cond, geom, None, cfg, detail=True)
    e, out = s["events"], s["out"]
    for k, v in cl[0].items():
        if k != "pulses":
            _keep(out, k, v, 512 + 2 * e)
    for k, v in cl[0]["pulses"].items():
        _keep(out, "pulse_" + k, v, 2000 + 200 * e)
    return out


def _synth_inputs(case, seed):
    """Charges of `channels` SiPMs: one or two bursts of about 30 PE within 60 ns each, in a 1.6 us window."""
    rng = np.random.default_rng(seed)
    n = case["channels"]
    bursts = 1 + (rng.random(n) < 0.4)
    lab = np.repeat(np.arange(n, dtype=np.int64) * 3 + 7, bursts)
    t0 = rng.uniform(20.0, 1500.0, len(lab))
    k = 1 + rng.poisson(28.0, len(lab))
    chan = np.repeat(lab, k)
    time = np.repeat(t0, k) + rng.exponential(9.0, len(chan))
    charge = 2.652e-13 * np.clip(rng.normal(1.0, 0.15, len(chan)), 0.05, None)
    o = np.lexsort((time, chan))
    tdc0 = rng.uniform(0.0, CF.PERIOD, 3 * n + 8)
    return chan[o], time[o], charge[o], tdc0


def _prepare_synth(case, seed):
    return {"in": _synth_inputs(case, seed), "cfg": CF.WaveformConfig(), "window": (0.0, 128 * CF.PERIOD),
            "rows": 2 * case["channels"], "out": {}}


def _run_synth(s):
    for k, v in WF.synthesize(*s["in"], s["cfg"], s["window"]).items():
        _keep(s["out"], k, v, s["rows"])
    return s["out"]


_KINDS = {"chain": (_prepare_chain, _run_chain), "fit": (_prepare_fit, _run_fit),
          "substeps": (_prepare_substeps, _run_substeps), "dropin": (_prepare_dropin, _run_dropin),
          "synth": (_prepare_synth, _run_synth)}


def prepare(case, seed):
    s = _KINDS[case["kind"]][0](case, seed)
    s["kind"] = case["kind"]
    return s


def run(state):
    return _KINDS[state["kind"]][1](state)


# ---- work and values --------------------------------------------------------------------------------------------

def work(case):
    """Bytes: inputs read once, outputs written once.  Operations: a keyed Philox block (60) and a logarithm per photon,
    three blocks per charge, the template sums of a charge's eight samples, and a fit of about 20 evaluations of eight
    samples (25 operations a sample) per pulse."""
    k = case["kind"]
    if k in ("chain", "dropin"):
        det = case.get("detector", "module")
        steps = case["events"] * _mean_steps(det)
        ph, ch, _, _, pu = PER_STEP[det]
        ops = steps * (80.0 * ph + 200.0 * ch + 4000.0 * pu)
        if det == "lookup":
            ops += steps * 4 * 198 * 60.0
        out = steps * (ch * 40 + pu * 150) if k == "dropin" else case["events"] * 0.05 * 200
        return {"bytes": 24.0 * steps + 28.0 * case["events"] + out, "flops": ops}
    if k == "fit":
        n = case["waveforms"]
        pulses = 5.0 * n
        return {"bytes": n * (195 * 2 + 44.0) + pulses * 104, "flops": pulses * 4000.0}
    if k == "substeps":
        n = case["rows"]
        return {"bytes": n * 144.0 + 137.0 * n * 24, "flops": n * 200 * 3 * 30.0 + 137.0 * n * 100}
    q = case["channels"] * 1.4 * 29
    return {"bytes": q * 24 + case["channels"] * 1.4 * 150, "flops": q * 16}


def exact(case, seed):
    """waveform.synthesize in plain NumPy (zero-suppressed digis of noiseless waveforms); None for the other kinds."""
    if case["kind"] != "synth":
        return None
    chan, time, charge, tdc0_of = _synth_inputs(case, seed)
    P, step, tmax, zs, thr = CF.PERIOD, 0.5, 100.0, 12, 5 * 0.0055
    z = (np.arange(0.0, tmax + step / 2, step) - 15.0) / 10.0
    tmpl = 0.0055 * np.e * np.exp(-z - np.exp(-z))
    tmpl = tmpl[:int(round(tmax / step))]                      # the template's grid ends below the maximum time
    new = np.r_[True, (chan[1:] != chan[:-1]) | (np.diff(time) > tmax + 4 * P)]
    cid, head = np.cumsum(new) - 1, np.flatnonzero(new)
    tail = np.r_[head[1:], len(chan)] - 1
    C = len(head)
    keep = (tail - head + 1) * tmpl.max() >= thr
    tdc0 = tdc0_of[chan[head]]
    ts = np.ceil((time[head] - P - tdc0) / P) * P + tdc0
    length = np.floor((time[tail] - time[head] + tmax) / P).astype(np.int64)
    j = np.maximum(np.ceil((time - ts[cid]) / P), 0).astype(np.int64)[:, None] + np.arange(int(tmax / P) + 3)
    dt = j * P + ts[cid][:, None] - time[:, None]
    ti = np.rint(dt / step).astype(np.int64)
    hit = (dt >= 0) & (ti < len(tmpl)) & keep[cid][:, None]
    row = np.broadcast_to(cid[:, None], j.shape)[hit]
    np.maximum.at(length, row, j[hit] + 1)
    width = int(length.max()) + zs
    wave = np.bincount(row * width + j[hit], (tmpl[np.minimum(ti, len(tmpl) - 1)]
                                              * (charge / 2.652e-13)[:, None])[hit], C * width).reshape(C, width)
    valid = np.arange(width) < length[:, None]
    over = (wave > thr) & valid
    near = over.copy()
    for d in (1, 2):
        near[:, :-d] |= over[:, d:]
        near[:, d:] |= over[:, :-d]
    near &= valid & keep[:, None]
    nxt, rows, cols = np.zeros(C, np.int64), [], []
    for i in range(width):
        start = ts + i * P
        r = np.flatnonzero(near[:, i] & (nxt <= i) & (start >= 0.0) & (start <= 128 * P))
        rows.append(r)
        cols.append(np.full(len(r), i))
        nxt[r] = i + zs
    r, c = np.concatenate(rows), np.concatenate(cols)
    start = ts[r] + c * P
    o = np.lexsort((start, chan[head][r]))
    r, c, start = r[o], c[o], start[o]
    at = c[:, None] + np.arange(zs)
    volt = np.where(at < length[r][:, None], wave[r[:, None], np.minimum(at, width - 1)], 0.0)
    out = {k: None for k in ("chan", "starttdc", "adc", "cluster_chan", "cluster_keep")}
    for k, v in (("start", start), ("tdc0", tdc0[r]), ("volt", volt), ("cluster_tstart", ts)):
        kept = {}
        _keep(kept, k, v, 2 * case["channels"])
        out.update(kept)
    return out
