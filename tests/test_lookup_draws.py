"""The lookup-table substeps' integer forms of FP64 rules (CPU), and table rows of every width and alignment on the GPU."""
from types import SimpleNamespace

import numpy as np
import pytest

from oracle import oracle as O


def ceil_uniform(k, total):
    """ceil(u * total) of u = k 2^-53, u * total rounded to FP64: as the device forms it from integers."""
    if total <= 0 or k == 0:
        return 0
    v = k * total
    s = v.bit_length() - 53
    if s > 0:
        rest, half = v & ((1 << s) - 1), 1 << (s - 1)
        v -= rest
        if rest > half or (rest == half and (v >> s) & 1):
            v += 1 << s
    return (v >> 53) + ((v & ((1 << 53) - 1)) != 0)


def test_integer_thresholds_equal_the_floating_point_ones():
    rng = np.random.default_rng(4)
    ks = [int(x) for x in rng.integers(0, 1 << 53, 3000)] + [0, 1, 2, (1 << 53) - 1, 1 << 52, (1 << 52) + 1]
    for total in (0, 1, 2, 3, 7, 255, 256, 1000, 4096, 38250, 65535, 1 << 20, (1 << 31) - 1):
        edge = []
        if total:
            for m in rng.integers(0, total, 40):         # uniforms whose product lies next to an integer
                e = (int(m) << 53) // total
                edge += [min((1 << 53) - 1, max(0, e + d)) for d in (-2, -1, 0, 1, 2)]
        for k in ks[:400] + ks[-6:] + edge:
            want = int(np.ceil(np.float64(k) * 2.0 ** -53 * np.float64(total)))
            assert ceil_uniform(k, total) == want, (k, total)


@pytest.mark.gpu
@pytest.mark.parametrize("ndelay,nemis", [(1, 1), (2, 3), (15, 16), (16, 17), (33, 8), (64, 5), (65, 64), (150, 8), (255, 2)])
def test_table_widths_bit_exact(ndelay, nemis):
    """FP64 photons equal the oracle's for delay and emission rows of any width (rows start at any byte, the first and
    last rows of a table included), with rows of zero weights; the FP32-mixed pass finds the same counts but for draws
    within rounding."""
    from crvgpu import lookup as LK
    rng = np.random.default_rng(ndelay * 7 + nemis)
    edges = {"x": np.linspace(0, 10, 3), "y": np.linspace(-26, 26, 4), "z": np.linspace(-1000, 1000, 3),
             "beta": np.linspace(0.4, 1, 3), "theta": np.linspace(0, np.pi, 3), "phi": np.linspace(0, np.pi, 3),
             "r": np.linspace(0, 0.7, 3)}

    def tab(n):
        d = rng.integers(0, 256, (n, ndelay)).astype(np.uint8)
        e = rng.integers(0, 9, (n, nemis)).astype(np.uint8)
        d[n // 2], e[n // 3] = 0, 0
        return SimpleNamespace(prob=rng.uniform(0, 0.05, n).astype(np.float32), delays=d,
                               delay_sum=d.sum(1, dtype=np.int32), emis=e, emis_sum=e.sum(1, dtype=np.int32))

    L = SimpleNamespace(half_thickness=9.64, half_width=25.42, half_length=1000.0, fiber_separation=26.0,
                        hole_radius_x=2.0, hole_radius_y=1.0, fiber_radius=0.7, corner_radius=1.75,
                        fiber_decay_time=2.0, edges=edges, tables={"scint": tab(12), "ckscint": tab(24), "ckfiber": tab(32)})
    R = 120
    a = np.c_[rng.uniform(-9.9, 9.9, R), rng.uniform(-25.9, 25.9, R), rng.uniform(-999, 999, R)]
    d = np.c_[rng.normal(0, 4, R), rng.normal(0, 4, R), rng.normal(0, 20, R)]
    k = np.arange(R) % 4 == 0                                  # through the fibres and along their hole's edge
    a[k, 0], a[k, 1] = rng.uniform(-2, 2, k.sum()), 13.0 * rng.choice([-1, 1], k.sum()) + rng.uniform(-1, 1, k.sum())
    d[k, :2] *= 0.1
    dl = np.linalg.norm(d, axis=1)
    t0 = rng.uniform(0, 1e3, R)
    rows = {"s": a, "d": d, "t0": t0, "t1": t0 + 0.1, "nsub": np.maximum((dl / 0.1).astype(np.int64), 1),
            "beta": rng.uniform(0.5, 1, R), "theta": np.arccos(np.clip(d[:, 2] / dl, -1, 1)), "dev": np.ones(R),
            "mu": rng.uniform(-2e-4, 2e-4, R) * (np.arange(R) % 3 > 0), "step": np.arange(R, dtype=np.int64),
            "chan": np.arange(R, dtype=np.int64) * 4, "n_scint": rng.integers(0, 60, R), "n_ck_s": rng.integers(0, 9, R),
            "n_ck_f": rng.integers(0, 20, R)}
    got = LK.substep_photons(L, rows, 5)
    want = O.substep_photons(L, rows, 5)
    assert not want[3] and len(want[0]) > 1000
    for g, w in zip(got, want):
        assert np.array_equal(g, w)
    n32 = np.bincount(LK.substep_photons(L, rows, 5, precision="fp32")[0], minlength=R)
    assert np.mean(n32 != np.bincount(got[0], minlength=R)) < 0.05
