"""FP32-mixed waveform settings beyond the fixed-point range (2^30 ns) are refused with CRV_ST_LIMIT: no digis, nothing
written, whatever the workspace held before."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("field,value", [("feb_phase_width", 3e9), ("spe_max_time", 2e9), ("period", float("nan"))])
@pytest.mark.parametrize("fill", (0x00, 0x01, 0xFF))
@pytest.mark.parametrize("caller_tdc0", (False, True))
def test_refused_settings_leave_no_digis(field, value, fill, caller_tdc0):
    import torch
    from crvgpu import _capi
    from crvgpu import config as CF
    from crvgpu import geometry as GM
    from crvgpu.params import make_params
    from crvgpu.response import DeviceTables
    from crvgpu.waveform import DIGI_KEYS, single_pe_template
    geom = GM.module_geometry(1)
    cfg = CF.ChainConfig(precision="fp32")
    T = DeviceTables(geom, GM.default_conditions(geom), cfg)
    tmpl = torch.from_numpy(single_pe_template(CF.WaveformConfig())).cuda()
    P = make_params(cfg, 3, template_len=int(tmpl.numel()))
    setattr(P, field, value)
    n, slots = 30000, 5000
    label = torch.arange(n, device="cuda") // 40 % 200 + torch.arange(n, device="cuda") // 8000 * 32768
    time = 100.0 + (torch.arange(n, device="cuda") % 40).double()
    charge = torch.full((n,), 2.652e-13, dtype=torch.float64, device="cuda")
    tdc0 = torch.zeros(n, dtype=torch.float64, device="cuda")
    L, zs = _capi.load(), int(P.samples_zs)
    size = L.crv_digis_workspace(ctypes.byref(P), n, slots)
    ws = torch.empty(size, dtype=torch.uint8, device="cuda").fill_(fill)
    kinds = dict(chan=torch.int64, start=torch.float64, tdc0=torch.float64, starttdc=torch.int64, volt=torch.float64,
                 adc=torch.int16)
    out = {k: torch.full((slots * (zs if k in ("volt", "adc") else 1),), 77, dtype=kinds[k], device="cuda")
           for k in DIGI_KEYS}
    D = _capi.CrvDigis(*[_capi.ptr(out[k]) for k in DIGI_KEYS])
    count = torch.full((1,), -1, dtype=torch.int64, device="cuda")
    st = _capi.DeviceStatus("cuda")
    tail = (slots, ctypes.byref(D), slots, _capi.ptr(count), _capi.ptr(ws), size,
            ctypes.c_void_p(torch.cuda.current_stream().cuda_stream), st.ptr)
    head = (ctypes.byref(P), ctypes.byref(T.c_channels()), n, _capi.ptr(label), _capi.ptr(time), _capi.ptr(charge))
    if caller_tdc0:
        rc = L.crv_synthesize(*head, _capi.ptr(tdc0), _capi.ptr(tmpl), int(tmpl.numel()), *tail)
    else:
        rc = L.crv_digis(*head, _capi.ptr(tmpl), int(tmpl.numel()), None, None, 0, *tail)
    _capi.check(rc, "digis")
    flags, need = st.read()
    assert flags == _capi.ST_LIMIT and int(count) == 0 and not np.any(need)
    for k, v in out.items():
        assert (v == 77).all(), k
