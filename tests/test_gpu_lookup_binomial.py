"""Arrival draws (a Binomial per substep) of the FP32-mixed lookup kernels where the first term of the inversion, (1 - p)^n, lies
below FP32's normal range: rows inside the scintillator, away from its hole and edges, in a table of one probability."""
from types import SimpleNamespace

import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _case(p, n_photons, rows=300, nsub=20):
    edges = {"x": np.linspace(0, 9.89, 4), "y": np.linspace(-25.67, 25.67, 4), "z": np.linspace(-1600, 1600, 5),
             "beta": np.linspace(0.455, 1.0, 3), "theta": np.linspace(0, np.pi, 4), "phi": np.linspace(0, np.pi, 4),
             "r": np.linspace(0, 0.616, 3)}
    nb = {k: len(v) - 1 for k, v in edges.items()}
    d = np.random.default_rng(2).integers(1, 9, 20, dtype=np.uint8)

    def table(m):
        return SimpleNamespace(prob=np.full(m, p, np.float32), delays=np.tile(d, (m, 1)),
                               delay_sum=np.full(m, int(d.sum()), np.int32), emis=np.ones((m, 2), np.uint8),
                               emis_sum=np.full(m, 2, np.int32))

    m = nb["x"] * nb["y"] * nb["z"]
    L = SimpleNamespace(name="t", edges=edges, half_thickness=9.64, half_width=25.42, half_length=1600.0,
                        fiber_separation=26.0, hole_radius_x=2.0, hole_radius_y=1.0, fiber_radius=0.7, corner_radius=1.75,
                        fiber_decay_time=0.0,
                        tables={"scint": table(m), "ckscint": table(m * nb["beta"]),
                                "ckfiber": table(nb["beta"] * nb["theta"] * nb["phi"] * nb["r"] * nb["z"])})
    rng = np.random.default_rng(3)
    one = np.ones(rows, np.int64)
    a = np.c_[np.full(rows, -4.0), rng.uniform(19, 20, rows), rng.uniform(-1500, 1500, rows)]
    dd = np.c_[np.full(rows, 8.0), rng.uniform(-0.5, 0.5, rows), rng.uniform(-0.5, 0.5, rows)]
    t0 = rng.uniform(0, 1e3, rows)
    return L, {"s": a, "d": dd, "t0": t0, "t1": t0 + 0.07, "nsub": nsub * one, "beta": np.full(rows, 0.999),
               "theta": np.full(rows, 1.5), "dev": np.ones(rows), "step": np.arange(rows), "chan": 0 * one,
               "n_scint": n_photons * one, "n_ck_s": 0 * one, "n_ck_f": 0 * one}


# (probability, photons per substep): means 90 to 255 and, at probabilities of 0.4 to 0.6, from 63 on
@pytest.mark.parametrize("p,n", [(2.0 ** -10, 100000), (2.0 ** -6, 5900), (2.0 ** -6, 16000), (0.125, 800), (0.25, 1000),
                                 (0.4375, 180), (0.5, 130), (0.5, 500), (0.5625, 200), (0.75, 900), (0.875, 1000)])
def test_fp32_draws_of_large_means_equal_the_oracles(p, n):
    """The probability is exact in FP32 and the draw is made in FP64 from the same words, so the counts are the oracle's
    but for the boundary of a substep's place, of which there is none here: every row's count, exactly."""
    from crvgpu import lookup as LK
    L, rows = _case(p, n)
    want = O.substep_photons(L, rows, 9)
    assert not want[3] and abs(len(want[0]) / (300 * 20 * n * p) - 1) < 0.01
    st, _, _ = LK.substep_photons(L, rows, 9, precision="fp32")
    assert np.array_equal(np.bincount(st, minlength=300), np.bincount(want[0], minlength=300))


@pytest.mark.parametrize("p,n", [(2.0 ** -11, 500), (0.0015, 486), (0.01, 60), (0.03, 900), (0.2, 3), (0.2, 500), (0.48, 40),
                                 (0.489, 170), (0.49, 40), (0.3, 420), (1e-5, 900000), (1.3e-4, 980000), (0.999, 30)])
def test_fp64_draws_decided_in_fp32_equal_the_oracles(p, n):
    """30,000 to 300,000 draws of each (probability, photons), from means of 0.24 to 127 at the ends of what FP32 decides: a
    comparison trusted wrongly moves a count or the photons behind it.  Bit for bit."""
    from crvgpu import lookup as LK
    nsub = 1000 if n * p < 20 else 100
    L, rows = _case(p, n, rows=300, nsub=nsub)
    want = O.substep_photons(L, rows, 21)
    assert not want[3] and len(want[0]) > 10000
    got = LK.substep_photons(L, rows, 21)
    for a, b in zip(got, want):
        assert np.array_equal(a, b)
