"""SiPM photons at -infinity and in the far past (crv_sipm takes any time): a pixel that fired then has recovered when it is hit
again.  FP64 against the oracle, bit for bit (whose fresh pixels fired at -infinity: finite times there); any time against
the same photons a millisecond earlier."""
from dataclasses import replace

import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _photons(early):
    """SiPMs of 40 to 1,100 photons on nine pixels, one of them at `early` (so most of the nine are hit again)."""
    rng = np.random.default_rng(4)
    n = np.array([40, 41, 100, 255, 256, 257, 600, 1100] * 6)
    label = np.repeat((1 << 20 | 9) * 32768 + np.arange(len(n), dtype=np.int64), n)
    t = rng.uniform(100, 900, len(label))
    first = np.cumsum(n) - n
    t[first] = early
    pmap = np.zeros((40, 40))
    pmap[5:8, 30:33] = 1.0
    return label, t, np.arange(len(label)) - np.repeat(first, n), pmap


@pytest.mark.parametrize("early", (-1e300, -1e30, -1e6))
def test_fp64_equals_the_oracle(early):
    from crvgpu.config import SiPMConfig
    from crvgpu.response import simulate
    label, t, key, pmap = _photons(early)
    sc = SiPMConfig()
    G = simulate(label, t, np.arange(len(label)), pmap, sc, None, t_end=1606.4, key=5, draw_key=key)
    Q, u, nq, nfp, st = O.sipm_groups(label, t, np.arange(len(label)), key, lambda L: np.zeros(len(L), np.int64), sc, 5,
                                      1606.4, pmap)
    assert st == 0 and np.count_nonzero(Q["time"] <= -1e5) > 10
    for c in ("chan", "time", "charge", "pe", "photon"):
        assert np.array_equal(G[c], Q[c]), c
    assert np.array_equal(G["_group_fired"], nfp) and np.array_equal(G["_group_charges"], nq)


@pytest.mark.parametrize("early", (-np.inf, -1e300, -1e30))
@pytest.mark.parametrize("precision", ("fp32", "fp64"))
def test_any_time_long_past_is_the_same(early, precision):
    """Without afterpulses, whose times are the photon's plus an interval."""
    from crvgpu.config import SiPMConfig
    from crvgpu.response import simulate
    sc = replace(SiPMConfig(), trap0_prob=0.0)
    out = []
    for e in (early, -1e6):
        label, t, key, pmap = _photons(e)
        out.append(simulate(label, t, np.arange(len(label)), pmap, sc, None, t_end=1606.4, key=5, draw_key=key,
                            precision=precision))
    late = out[0]["time"] > 0
    assert np.array_equal(late, out[1]["time"] > 0) and np.count_nonzero(~late) > 10
    assert np.array_equal(out[0]["time"][late], out[1]["time"][late])
    for c in ("chan", "charge", "pe", "photon", "_group_fired", "_group_charges"):
        assert np.array_equal(out[0][c], out[1][c]), c
