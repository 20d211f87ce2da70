"""Scratch of the prefix sums on both sides of 155,648 items, where tiles of one item per thread (304 of them) end and tiles
of eight (39 of them) begin: a scratch sized for more items serves any smaller sum.  Batches with more events than
steps sum over both in one scratch."""
import ctypes

import numpy as np
import pytest

EDGES = [4096, 4097, 155648, 155649, 156000, 400000, 155648 * 8, 155648 * 8 + 1, 3000000]


def test_workspaces_grow_with_their_counts():
    from crvgpu import _capi
    from crvgpu.params import make_params
    L, P = _capi.load(), make_params()
    for f in (L.crv_reco_waveforms_workspace, L.crv_pulse_hits_workspace, L.crv_lookup_rows_workspace,
              lambda n: L.crv_coincidences_workspace(n, 1000),
              lambda n: L.crv_response_workspace(ctypes.byref(P), n, 1000, 1000, 8),
              lambda n: L.crv_response_workspace(ctypes.byref(P), 10, n // 4, 1000, 8)):
        sizes = [f(n) for n in EDGES]
        assert sizes == sorted(sizes) and sizes[0] > 0


def test_one_scratch_serves_every_smaller_sum():
    """From the sizes alone: a waveform workspace is 16-word totals and padding beyond its sum's scratch, which is two words
    for each tile of any smaller sum at least."""
    from crvgpu import _capi
    L = _capi.load()
    tiles = lambda n: -(-n // 512) if 4096 < n <= 155648 else -(-n // 4096)  # noqa: E731
    for n in EDGES:
        words = L.crv_reco_waveforms_workspace(n) // 8
        assert words >= 2 * max(tiles(m) for m in EDGES if m <= n) + 8


# events, steps: the events' sum in small tiles and the SiPMs' in large ones, and the other way round
SPARSE = [(100000, 40000), (65536, 40000), (200000, 25000), (155649, 300), (155648, 38912)]


@pytest.mark.gpu
@pytest.mark.parametrize("ne,ns", SPARSE)
def test_more_events_than_steps(ne, ns):
    """Events without steps change nothing: the charges of a batch with and without them are the same."""
    import torch
    from crvgpu import config as CF
    from crvgpu import geometry as GM
    from crvgpu.params import make_params
    from crvgpu.response import DeviceSteps, DeviceTables, engine, upload_steps
    geom = GM.module_geometry()
    cond, cfg = GM.default_conditions(geom), CF.ChainConfig(precision="fp32")
    steps = GM.synthetic_steps(max(1, ns // 40), geom, seed=ne)
    m = min(ns, len(steps["edep"]))
    steps = {k: np.asarray(v)[:m] for k, v in steps.items()}
    few = upload_steps(steps, nbars=geom.nbars)
    P = make_params(cfg, 5, uniform_map=True)
    T = DeviceTables(geom, cond, cfg)
    want = engine().run(P, few, T)
    # the same events at places of their own among ne
    rng = np.random.default_rng(ne)
    at = np.sort(rng.choice(ne, few.nevents, replace=False))
    key = few.ev_event.cpu().numpy()
    dev = few.x.device

    def spread(col, fill):
        out = np.asarray(fill).astype(col.cpu().numpy().dtype)
        out[at] = col.cpu().numpy()
        return torch.from_numpy(out).to(dev)

    assert np.all(np.diff(key) > 0)
    first = np.append(few.ev_first.cpu().numpy(), m)[np.searchsorted(at, np.arange(ne))]
    zero = np.zeros(ne)
    many = DeviceSteps(x=few.x, y=few.y, z=few.z, t=few.t, edep=few.edep, bar=few.bar,
                       ev_event=spread(few.ev_event, zero), ev_subrun=spread(few.ev_subrun, zero),
                       ev_run=spread(few.ev_run, zero), ev_first=spread(few.ev_first, first),
                       ev_nsteps=spread(few.ev_nsteps, zero), nsteps=few.nsteps, nevents=ne, max_steps=few.max_steps)
    got = engine().run(P, many, T)
    assert got.n == want.n > 1000 and got.nsipm == want.nsipm
    for k in ("label", "time", "charge", "pe", "photon", "sipm_label", "sipm_photons", "sipm_fired"):
        assert torch.equal(getattr(got, k), getattr(want, k)), k


@pytest.mark.gpu
def test_waveforms_in_a_workspace_of_a_larger_count():
    import torch
    from crvgpu import _capi, config as CF, geometry as GM
    from crvgpu.chain import ChainEngine
    geom = GM.module_geometry(1)
    eng = ChainEngine(geom, GM.default_conditions(geom), CF.ChainConfig())
    L, P, n = _capi.load(), eng.params(1), 100000
    size = L.crv_reco_waveforms_workspace(200000)
    label = torch.arange(n, device="cuda") // 7 % 1000 + torch.arange(n, device="cuda") // 7000 * 32768
    tdc = torch.arange(n, device="cuda") * P.samples_zs
    i64, f64 = (lambda: torch.zeros(n, dtype=torch.int64, device="cuda")), \
        (lambda: torch.zeros(n, dtype=torch.float64, device="cuda"))
    out = [i64(), i64(), torch.zeros(n, dtype=torch.int32, device="cuda"), i64(), f64(), f64(), f64(), f64()]
    count, st = torch.zeros(1, dtype=torch.int64, device="cuda"), torch.zeros(64, dtype=torch.int64, device="cuda")
    ws = torch.empty(size + 4096, dtype=torch.uint8, device="cuda").fill_(0x5A)
    _capi.check(L.crv_reco_waveforms(ctypes.byref(P), ctypes.byref(eng.tabs.c_channels()), n, _capi.ptr(label),
                                     _capi.ptr(tdc), *[_capi.ptr(v) for v in out], _capi.ptr(count), _capi.ptr(ws),
                                     size, torch.cuda.current_stream().cuda_stream, _capi.ptr(st)), "crv_reco_waveforms")
    start = torch.nonzero(torch.cat([torch.ones(1, dtype=torch.bool, device="cuda"), label[1:] != label[:-1]])).ravel()
    assert int(count) == len(start) and torch.equal(out[1][:len(start)], start * P.samples_zs)
    assert (ws[size:] == 0x5A).all()
