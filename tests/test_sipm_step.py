"""The SiPM stage's photon step: draws decided on integers (CPU), and the step's edges against the oracle (GPU)."""
from dataclasses import replace

import numpy as np
import pytest

from oracle import oracle as O


def test_pixel_bin_and_draw_thresholds_equal_the_floating_point_rules():
    """floor(u * 1600) by integers equals the FP64 product's floor, also where the product rounds up to an integer; and
    bits < T decides uni < q as the floating-point compare does."""
    rng = np.random.default_rng(3)
    M = (1 << 53) - 1
    k = [int(v) for v in rng.integers(0, 1 << 53, 4000)] + [0, 1, M]
    for b in rng.integers(1, 1600, 1500):                # draws next to the edges of a bin
        e = (int(b) << 47) // 25
        k += [min(M, max(0, e + d)) for d in range(-3, 4)]
    for v in k:
        m = v * 25
        b = m >> 47
        s = m.bit_length() - 53
        if s > 0 and (m & ((1 << 47) - 1)) >= (1 << 47) - (1 << (s - 1)):
            b += 1
        assert b == int(np.floor(np.float64(v) * 2.0 ** -53 * 1600.0)), v
    for bits, dt in ((53, np.float64), (24, np.float32)):
        one = dt(2.0 ** bits)
        for q in [dt(x) for x in rng.random(300)] + [dt(0), dt(1), dt(-0.5), dt(2), dt(np.nan), dt(1e-300), dt(2.0 ** -bits)]:
            x = q * one
            T = 0 if not x > 0 else (1 << bits) if x >= one else int(x) + (1 if dt(int(x)) < x else 0)
            at = int(x) if np.isfinite(x) else 0
            for v in {0, 1, max(0, at - 1), max(0, at), at + 1, (1 << bits) - 1}:
                if 0 <= v < 1 << bits:
                    assert (v < T) == bool(dt(v) * dt(2.0 ** -bits) < q), (bits, v, q)


@pytest.mark.gpu
@pytest.mark.parametrize("pixel_id", ["truncate", "lrint"])
@pytest.mark.parametrize("where", ["everywhere", "block"])
@pytest.mark.parametrize("cross_talk", [0.0, 0.05, 0.25])
def test_step_edges_bit_exact(pixel_id, where, cross_talk):
    """SiPMs of 1 photon up to the passes' capacities, photons in order and out of order, on the whole map or on a block
    of nine bins (every touch then meets pixels that earlier photons and cross-talk nodes of its step touch)."""
    from crvgpu.config import SiPMConfig
    from crvgpu.response import simulate
    rng = np.random.default_rng(17)
    pmap = np.ones((40, 40))
    if where == "block":
        pmap[:] = 0.0
        pmap[5:8, 30:33] = 1.0
    sizes = [1, 2, 31, 32, 33, 63, 64, 65, 96, 255, 256, 257, 700, 1024, 1025, 2500, 4096]
    if where == "everywhere":
        sizes += [int(v) for v in rng.integers(1, 260, 200)]
    n = np.array(sizes * 2)
    label = np.repeat((1 << 20 | 9) * 32768 + np.arange(len(n), dtype=np.int64), n)
    t = np.repeat(rng.uniform(0, 800, len(n)), n) + rng.exponential(20.0, len(label))
    half = label >= label[sum(sizes)]                    # the second half of the SiPMs in time order
    o = np.lexsort((np.where(half, t, 0.0), label))
    t = t[o]
    sc = replace(SiPMConfig(pixel_id=pixel_id), cross_talk=cross_talk)
    key = np.arange(len(label)) - np.repeat(np.cumsum(n) - n, n)
    G = simulate(label, t, np.arange(len(label)), pmap, sc, None, t_end=1606.4, key=5, draw_key=key)
    Qo, u, nq, nfp, st = O.sipm_groups(label, t, np.arange(len(label)), key, lambda L: np.zeros(len(L), np.int64), sc, 5,
                                       1606.4, pmap)
    assert st == 0
    for c in ("chan", "time", "charge", "pe", "photon"):
        assert np.array_equal(G[c], Qo[c]), c
    assert np.array_equal(G["_group_fired"], nfp) and np.array_equal(G["_group_charges"], nq)


@pytest.mark.gpu
@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_charge_factor_takes_the_time_per_pixel_pass(precision):
    """More charge slots per photon (charge_factor) send every SiPM to the passes that keep a time per pixel: same charges
    as the first pass's times per record."""
    from crvgpu import response as R
    from crvgpu.params import make_params
    from tests.helpers import workload
    geom, cond, cfg, steps = workload(40, seed=8)
    cfg.precision = precision
    ds, tabs = R.upload_steps(steps, nbars=geom.nbars), R.DeviceTables(geom, cond, cfg)
    out = []
    for factor in (1, 3):
        P = make_params(cfg, 9, charge_factor=factor)
        r = R.ResponseEngine().run(P, ds, tabs)
        out.append([getattr(r, k).cpu().numpy() for k in ("label", "time", "charge", "pe", "photon")])
    assert len(out[0][0]) > 1000
    for a, b in zip(*out):
        assert np.array_equal(a, b)
