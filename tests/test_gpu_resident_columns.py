"""A batch's columns into the resident chain's buffers and its clusters out of them in one launch, against the copies
column by column: sizes around the 16-byte words, slices off their alignment, and the columns the one launch does not
take (other types, strides, host memory).  Exact."""
from dataclasses import replace

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _chain(events, steps):
    from crvgpu import config as CF
    from crvgpu import geometry as GM
    from crvgpu.chain import ChainEngine
    from crvgpu.resident import ChainCaps, ResidentChain
    geom = GM.module_geometry(1)
    eng = ChainEngine(geom, GM.default_conditions(geom), CF.ChainConfig())
    return ResidentChain(eng, ChainCaps(events=events, steps=steps, photons=1000, charges=1000, slots=1000, digis=1000,
                                        pulses=1000, max_steps_per_event=200), graph=False)


def _steps(e, n, cut, rng):
    import torch
    from crvgpu.response import DeviceSteps
    f = lambda m, dt, lo=-2 ** 31: torch.from_numpy(  # noqa: E731
        rng.integers(lo, 2 ** 31 - 1, m + cut).astype(dt)).cuda()[cut:]
    cols = [f(n, np.float32) for _ in range(5)] + [f(n, np.int32)] + [f(e, np.int32) for _ in range(3)]
    return DeviceSteps(*cols, ev_first=f(e, np.int64), ev_nsteps=f(e, np.int32), nsteps=n, nevents=e, max_steps=7)


def _state(rc):
    return {k: v.cpu().numpy().copy() for d in (rc.st, rc.ev, {"n": rc.nsteps_dev}) for k, v in d.items()}


@pytest.mark.parametrize("cut", (0, 1, 3, 4))
@pytest.mark.parametrize("e,n", [(0, 0), (1, 1), (3, 5), (15, 33), (16, 4097), (64, 300000)])
def test_load(e, n, cut):
    rc = _chain(64, 300000)
    ds = _steps(e, n, cut, np.random.default_rng(7 * n + cut))
    rc._load_each(ds, None)
    want = _state(rc)
    for k, v in rc.st.items():
        v[:n].fill_(5)
    for k, v in rc.ev.items():                # rows beyond the batch: key, first and nsteps are cleared, the rest stay
        v[:None if k in ("key", "first", "nsteps") else e].fill_(5)
    assert rc._load_columns(ds, None)
    got = _state(rc)
    assert all(np.array_equal(got[k], want[k]) for k in want)


def test_columns_of_other_forms_are_copied_one_by_one():
    import torch
    rc = _chain(8, 64)
    ds = _steps(5, 40, 0, np.random.default_rng(1))
    rc.load(ds)
    want = _state(rc)
    forms = [replace(ds, ev_nsteps=ds.ev_nsteps.to(torch.int64)), replace(ds, bar=ds.bar.to(torch.int64)),
             replace(ds, y=torch.stack([ds.y, ds.y], 1)[:, 0]), replace(ds, ev_run=ds.ev_run.cpu())]
    for other in forms:
        assert not rc._load_columns(other, None)
        rc.load(other)
        got = _state(rc)
        assert all(np.array_equal(got[k], want[k]) for k in want)
    with pytest.raises(RuntimeError):
        rc.load(replace(ds, z=ds.z[:-1]))


@pytest.mark.parametrize("ncl,nm", [(0, 0), (0, 3), (1, 0), (1, 2), (5, 17), (999, 1000)])
def test_take(ncl, nm):
    import torch
    rc = _chain(8, 64)
    for d in (rc.cl, rc.mem):
        for v in d.values():
            v.copy_(torch.randint(0, 200, v.shape, device="cuda").to(v.dtype))
    cl, mem = rc._take(ncl, nm)
    for d, got, n in ((rc.cl, cl, ncl), (rc.mem, mem, nm)):
        assert list(got) == list(d)
        for k, v in d.items():
            assert got[k].dtype == v.dtype and got[k].shape == v[:n].shape and torch.equal(got[k], v[:n])
            assert n == 0 or got[k].data_ptr() != v.data_ptr()
