"""FP32-mixed groups with a charge time beyond the fixed-point range (2^30 ns, infinities, NaN) report CRV_ST_LIMIT and give no
digis, at once for short sampling periods too; the groups beside them give the digis that they give without them."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _digis(P, T, tmpl, label, time, charge):
    import torch
    from crvgpu import _capi
    from crvgpu.waveform import DIGI_KEYS
    L, zs, n, slots = _capi.load(), int(P.samples_zs), len(label), 40000
    up = lambda a, t: torch.from_numpy(np.ascontiguousarray(np.asarray(a, t))).cuda()  # noqa: E731
    cols = [up(label, np.int64), up(time, np.float64), up(charge, np.float64)]
    ws = torch.zeros(L.crv_digis_workspace(ctypes.byref(P), n, slots), dtype=torch.uint8, device="cuda")
    kinds = dict(chan=torch.int64, start=torch.float64, tdc0=torch.float64, starttdc=torch.int64, volt=torch.float64,
                 adc=torch.int16)
    out = {k: torch.zeros(slots * (zs if k in ("volt", "adc") else 1), dtype=kinds[k], device="cuda") for k in DIGI_KEYS}
    D = _capi.CrvDigis(*[_capi.ptr(out[k]) for k in DIGI_KEYS])
    count, st = torch.zeros(1, dtype=torch.int64, device="cuda"), _capi.DeviceStatus("cuda")
    _capi.check(L.crv_digis(ctypes.byref(P), ctypes.byref(T.c_channels()), n, *[_capi.ptr(c) for c in cols],
                            _capi.ptr(tmpl), int(tmpl.numel()), None, None, 0, slots, ctypes.byref(D), slots,
                            _capi.ptr(count), _capi.ptr(ws), ws.numel(),
                            ctypes.c_void_p(torch.cuda.current_stream().cuda_stream), st.ptr), "crv_digis")
    m = int(count)
    return st.read()[0], {k: v[:m * (zs if k in ("volt", "adc") else 1)].cpu().numpy() for k, v in out.items()}


@pytest.mark.parametrize("period", (12.55, 0.75))
@pytest.mark.parametrize("far", (np.nan, np.inf, -np.inf, 1.2e9, -1.2e9, 1e300))
@pytest.mark.parametrize("where", ("first", "middle", "last", "all"))
def test_far_times_drop_their_group_alone(far, where, period):
    import torch
    from crvgpu import _capi
    from crvgpu import config as CF
    from crvgpu import geometry as GM
    from crvgpu.params import make_params
    from crvgpu.response import DeviceTables
    from crvgpu.waveform import single_pe_template
    geom, cfg = GM.module_geometry(1), CF.ChainConfig(precision="fp32")
    T = DeviceTables(geom, GM.default_conditions(geom), cfg)
    tmpl = torch.from_numpy(single_pe_template(CF.WaveformConfig())).cuda()
    P = make_params(cfg, 3, template_len=int(tmpl.numel()))
    P.period, P.noise_on = period, 0
    groups, k = 150, 30
    label = np.repeat(np.arange(groups), k)
    time = 100.0 + 5.0 * (label % 7) + np.tile(np.arange(k), groups)
    charge = np.full(len(label), 2.652e-13)
    bad = np.isin(label, (3, 4, 40, 149))
    good = _digis(P, T, tmpl, label[~bad], time[~bad], charge[~bad])
    assert good[0] == 0 and len(good[1]["chan"]) >= groups - 4
    at = np.tile(np.arange(k), groups)
    pick = bad & {"first": at == 0, "middle": at == k // 2, "last": at == k - 1, "all": at >= 0}[where]
    time[pick] = far
    flags, got = _digis(P, T, tmpl, label, time, charge)
    assert flags == _capi.ST_LIMIT
    for c in got:
        assert np.array_equal(got[c], good[1][c]), c
