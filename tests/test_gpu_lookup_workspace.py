"""Lookup photons in workspaces from the least that is accepted (no arrival counts kept) to the whole (counts of 256 substeps a
row kept): the same photons, and nothing written behind the workspace; less is refused."""
import ctypes

import numpy as np
import pytest

from tests.test_oracle_lookup import lookup_fixture

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ("fp32", "fp64"))
@pytest.mark.parametrize("n", (1, 3, 500))
def test_any_workspace_gives_the_same_photons(precision, n):
    import torch
    from crvgpu import _capi
    from crvgpu import lookup as LK
    table, rows, _ = lookup_fixture()
    D, R = LK.DeviceLookup(table), LK.DeviceRows({k: np.array(v)[40:40 + n] for k, v in rows.items()})
    L, S, C = _capi.load(), D.c(precision), R.c()
    whole, cap = L.crv_substeps_workspace(n), 300 * n + 4096
    least = whole - 512 * n
    want = None
    for size in (whole, whole + 777, whole - 1, whole - 64 * n, least + 256 * n, least + 64 * n, least + 64 * n - 1, least + 1, least):
        ws = torch.full((size + 4096,), 0xA5, dtype=torch.uint8, device="cuda")
        out = [torch.zeros(cap, dtype=t, device="cuda") for t in (torch.int64, torch.int64, torch.float64)]
        count, st = torch.zeros(1, dtype=torch.int64, device="cuda"), _capi.DeviceStatus("cuda")

        def call(nbytes):
            return L.crv_substep_photons(ctypes.byref(S), ctypes.c_uint32(5), ctypes.byref(C), n,
                                         *[_capi.ptr(o) for o in out], cap, _capi.ptr(count), _capi.ptr(ws), nbytes,
                                         ctypes.c_void_p(torch.cuda.current_stream().cuda_stream), st.ptr)
        _capi.check(call(size), "crv_substep_photons")
        assert st.read()[0] == 0 and (ws[size:] == 0xA5).all()
        got = [o[:int(count)].clone() for o in out]
        want = want or got
        assert len(got[0]) > 0 and all(torch.equal(a, b) for a, b in zip(got, want)), size
    assert call(least - 1) == _capi.CRV_ERR_ARG
