"""Rows of runs as the engine's prefix sums place them, at the sizes where the sums change their form: one tile (4,096
items), tiles of one item per thread, tiles that add up their predecessors, tiles after a scan of the tile sums (over
2,048 tiles).  Whole numbers and copied values: exact."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
SIZES = [(1, 1), (31, 2), (4095, 3), (4096, 1), (4097, 40), (8192, 5000), (155648, 90), (155649, 90), (4096 * 513 + 1, 7), (4096 * 2048, 2),
         (4096 * 2048 + 1, 90000), (4096 * 4097 + 33, 3)]


def _engine():
    from crvgpu import config as CF
    from crvgpu import geometry as GM
    from crvgpu.chain import ChainEngine
    geom = GM.module_geometry(1)
    return geom, ChainEngine(geom, GM.default_conditions(geom), CF.ChainConfig())


def _runs(n, mean):
    rng = np.random.default_rng(n)
    head = rng.random(n) < 1.0 / mean
    head[0] = True
    return rng, np.cumsum(head) - 1, np.flatnonzero(head)


def _dev(a, dt=np.int64):
    import torch
    return torch.from_numpy(np.ascontiguousarray(a, dt)).cuda()


@pytest.mark.parametrize("n,mean", SIZES)
def test_waveform_rows(n, mean):
    import torch
    from crvgpu import _capi
    geom, eng = _engine()
    _, run, start = _runs(n, mean)
    label = run // 2 * 32768 + run // 2 % (4 * geom.nbars)       # every second run: the same label after a gap
    L, P = _capi.load(), eng.params(1)
    tdc = 100 * run + P.samples_zs * (np.arange(n) - start[run])
    tdc += (run > 0) * 7
    d_lab, d_tdc = _dev(label), _dev(tdc)
    out = {k: torch.full((n,), -1, dtype=dt, device="cuda") for k, dt in
           (("label", torch.int64), ("off", torch.int64), ("n", torch.int32), ("start", torch.int64),
            ("ped", torch.float64), ("area", torch.float64), ("height", torch.float64), ("toff", torch.float64))}
    count = torch.full((1,), -1, dtype=torch.int64, device="cuda")
    st = torch.zeros(64, dtype=torch.int64, device="cuda")
    ws = torch.empty(int(L.crv_reco_waveforms_workspace(n)), dtype=torch.uint8, device="cuda")
    _capi.check(L.crv_reco_waveforms(ctypes.byref(P), ctypes.byref(eng.tabs.c_channels()), n, _capi.ptr(d_lab),
                                     _capi.ptr(d_tdc), *[_capi.ptr(v) for v in out.values()], _capi.ptr(count),
                                     _capi.ptr(ws), ws.numel(), torch.cuda.current_stream().cuda_stream,
                                     _capi.ptr(st)), "crv_reco_waveforms")
    m = int(count)
    joins = (np.diff(label) == 0) & (np.diff(tdc) == P.samples_zs)
    start = np.flatnonzero(np.append(True, ~joins))
    assert m == len(start)
    want = {"label": label[start], "off": start * P.samples_zs, "n": np.diff(np.append(start, n)) * P.samples_zs,
            "start": tdc[start]}
    for k, v in want.items():
        got = out[k].cpu().numpy()
        assert np.array_equal(got[:m], v) and (got[m:] == -1).all(), k


@pytest.mark.parametrize("ignore", (0, 1))
@pytest.mark.parametrize("n,mean", SIZES[:10])
def test_hits_and_events(n, mean, ignore):
    import torch
    from crvgpu import _capi
    geom, eng = _engine()
    rng, run, _ = _runs(n, mean)
    chan = rng.integers(0, 4 * geom.nbars, n)
    label = run * 32768 + chan
    status = rng.integers(0, 4, 4 * geom.nbars)
    L, P = _capi.load(), eng.params(1)
    P.ignore_channels, P.use_time_offset_db = ignore, 0
    t, pe, seq = rng.random(n), rng.random(n), rng.integers(0, 9, n)
    cols = [_dev(status, np.int32), _dev(label), _dev(np.zeros(n), np.float64), _dev(np.arange(n)), _dev(seq),
            _dev(t, np.float64), _dev(pe, np.float64)]
    out = {k: torch.full((n,), -1, dtype=dt, device="cuda") for k, dt in
           (("ev_start", torch.int64), ("ev_count", torch.int32), ("ev_key", torch.int64), ("bar", torch.int32),
            ("sipm", torch.int32), ("seq", torch.int32), ("time", torch.float64), ("pe", torch.float64))}
    nn = torch.full((2,), -1, dtype=torch.int64, device="cuda")
    st = torch.zeros(64, dtype=torch.int64, device="cuda")
    ws = torch.empty(int(L.crv_pulse_hits_workspace(n)), dtype=torch.uint8, device="cuda")
    c = [_capi.ptr(v) for v in cols]
    _capi.check(L.crv_pulse_hits(ctypes.byref(P), c[0], n, c[1], c[2], None, n, c[3], c[4], c[5], c[6],
                                 *[_capi.ptr(v) for v in out.values()], _capi.ptr(nn[0:1]), _capi.ptr(nn[1:2]),
                                 _capi.ptr(ws), ws.numel(), torch.cuda.current_stream().cuda_stream, _capi.ptr(st)),
                "crv_pulse_hits")
    kept = (status[chan] & 2 == 0) if ignore else np.ones(n, bool)
    ev = run[kept]
    start = np.flatnonzero(np.diff(ev, prepend=-1))
    want = {"ev_start": start, "ev_count": np.diff(np.append(start, len(ev))), "ev_key": ev[start],
            "bar": chan[kept] // 4, "sipm": chan[kept] % 4, "seq": seq[kept], "time": t[kept], "pe": pe[kept]}
    assert nn.tolist() == [len(start), len(ev)]
    for k, v in want.items():
        got = out[k].cpu().numpy()
        assert np.array_equal(got[:len(v)], v) and (got[len(v):] == -1).all(), k
