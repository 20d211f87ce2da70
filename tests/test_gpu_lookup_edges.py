"""FP32-mixed lookup tables of up to 48 KB of bin edges (they lie in shared memory, beside the emission's queues from 38.25 KB
on through the kernel's opt-in).  Every bin of a table holds the same entries, so more bins change nothing: the photons
are exactly those of the same table with few bins.  More edges than that stay refused."""
from types import SimpleNamespace

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
REST = 4 + 4 + 3 + 4 + 4 + 3 + 4 + 4        # edges other than z's: x, y, beta, theta, phi, r and the cosines of phi and theta


def _table(nz, like=None):
    edges = {"x": np.linspace(0, 9.89, 4), "y": np.linspace(-25.67, 25.67, 4), "z": np.linspace(-1600, 1600, nz + 1),
             "beta": np.linspace(0.455, 1.0, 3), "theta": np.linspace(0, np.pi, 4), "phi": np.linspace(0, np.pi, 4),
             "r": np.linspace(0, 0.616, 3)}
    nb = {k: len(v) - 1 for k, v in edges.items()}
    rng = np.random.default_rng(2)
    d, e = rng.integers(0, 9, 20, dtype=np.uint8), rng.integers(1, 40, 8, dtype=np.uint8)

    def table(m, p):
        return SimpleNamespace(prob=np.full(m, p, np.float32), delays=np.tile(d, (m, 1)),
                               delay_sum=np.full(m, int(d.sum()), np.int32), emis=np.tile(e, (m, 1)),
                               emis_sum=np.full(m, int(e.sum()), np.int32))

    m = nb["x"] * nb["y"] * nb["z"]
    tables = {"scint": table(m, 0.0015), "ckscint": table(m * nb["beta"], 0.002),
              "ckfiber": table(nb["beta"] * nb["theta"] * nb["phi"] * nb["r"] * nb["z"], 0.01)}
    geo = dict(half_thickness=9.64, half_width=25.42, half_length=1600.0, fiber_separation=26.0, hole_radius_x=2.0,
               hole_radius_y=1.0, fiber_radius=0.7, corner_radius=1.75, fiber_decay_time=7.4)
    if like is not None:
        geo.update({k: getattr(like, k) for k in geo})
    return SimpleNamespace(name="t", edges=edges, tables=tables, **geo)


def _rows(n=400):
    rng = np.random.default_rng(5)
    a = np.c_[np.full(n, -10.0), rng.uniform(-24, 24, n), rng.uniform(-1500, 1500, n)]
    d = np.c_[np.full(n, 20.0), rng.normal(0, 2, n), rng.normal(0, 2, n)]
    t0, one = rng.uniform(0, 1e5, n), np.ones(n, np.int64)
    return {"s": a, "d": d, "t0": t0, "t1": t0 + 0.07, "nsub": 200 * one, "beta": np.full(n, 0.999),
            "theta": np.full(n, 1.5), "dev": np.full(n, 0.94), "step": np.arange(n), "chan": 4 * np.arange(n),
            "n_scint": 480 * one, "n_ck_s": 30 * one, "n_ck_f": 30 * one}


def _photons(L, precision):
    from crvgpu import lookup as LK
    return [x.cpu().numpy() for x in LK.SubstepEngine().run(LK.DeviceLookup(L), LK.DeviceRows(_rows()), 7,
                                                            precision=precision)]


@pytest.mark.parametrize("nbytes", (39168, 39172, 44000, 49148, 49152))
def test_edges_up_to_48_kb(nbytes):
    want = _photons(_table(10), "fp32")
    assert len(want[0]) > 20000
    got = _photons(_table(nbytes // 4 - REST - 1), "fp32")
    for a, b in zip(got, want):
        assert np.array_equal(a, b)


def test_more_edges_are_refused_in_fp32_alone():
    big = _table(49156 // 4 - REST - 1)
    with pytest.raises(ValueError):
        _photons(big, "fp32")
    want = _photons(_table(10), "fp64")
    for a, b in zip(_photons(big, "fp64"), want):
        assert np.array_equal(a, b)


def test_chain_with_44_kb_of_edges():
    """The same inside a captured chain: the clusters' inputs are the charges, whose photons the table gives."""
    import torch
    from crvgpu.chain import ChainEngine
    from crvgpu.config import ChainConfig
    from crvgpu.lookup import LookupModel
    from crvgpu.resident import ChainCaps, ResidentChain
    from crvgpu.response import upload_steps
    from tests.helpers import module_lookup
    geom, cond, tables, lcfg, steps, pdg = module_lookup(60, seed=4)
    (name, base), = tables.items()
    counts = []
    for nz in (10, 44000 // 4 - REST - 1):
        L = _table(nz, like=base)
        L.edges["z"] = np.linspace(-base.half_length, base.half_length, nz + 1)
        L.name, L.reflector, L.ck_scint, L.ck_fiber = name, base.reflector, base.ck_scint, base.ck_fiber
        cfg = ChainConfig(lookup=lcfg, precision="fp32")
        model = LookupModel(geom, lcfg, {name: L}, cond.deviation, precision="fp32")
        ds, cols = upload_steps(steps, nbars=geom.nbars), model.upload_steps(steps, pdg)
        big = 400 * ds.nsteps + 4096
        caps = ChainCaps(events=ds.nevents, steps=ds.nsteps, photons=big, charges=big, slots=big, digis=big, pulses=big,
                         max_steps_per_event=ds.max_steps)
        rc = ResidentChain(ChainEngine(geom, cond, cfg), caps, real_dtype=torch.float64, graph=True, grow=True, max_grow=8,
                           lookup=model)
        counts.append(rc.run(ds, 21, lookup_steps=cols).counts)
    assert counts[0]["photons"] > 1000
    assert counts[0] == counts[1]
