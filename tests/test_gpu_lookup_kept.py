"""Photons of rows whose substeps' arrival counts the emission draws again: rows of more substeps than are kept (256), and
substeps of 255 arrivals and more, among ordinary ones.  FP64 against the oracle, bit for bit; FP32-mixed against
the same rows each in a batch of its own."""
import numpy as np
import pytest

from oracle import oracle as O
from tests.test_oracle_lookup import lookup_fixture

pytestmark = pytest.mark.gpu


def _rows(kind):
    L, rows, _ = lookup_fixture()
    n = len(rows["nsub"])
    pick = np.arange(n) % 7
    rows = {k: np.array(v) for k, v in rows.items()}
    if kind in ("long", "both"):
        rows["nsub"] = np.where(pick == 2, 255 + np.arange(n) % 4, np.where(pick == 5, 700, rows["nsub"]))
    if kind in ("dense", "both"):
        for k in ("n_scint", "n_ck_s", "n_ck_f"):
            rows[k] = np.where(pick % 3 == 1, rows[k] * 60 + 400, rows[k])
    cut = slice(0, 120)
    return L, {k: v[cut] for k, v in rows.items()}


@pytest.mark.parametrize("kind", ("long", "dense", "both"))
def test_fp64_equals_the_oracle(kind):
    from crvgpu import lookup as LK
    L, rows = _rows(kind)
    st, ch, tm = LK.substep_photons(L, rows, 9)
    ost, och, otm, lim = O.substep_photons(L, rows, 9)
    assert not lim and len(st) > 1000
    assert np.array_equal(st, ost) and np.array_equal(ch, och) and np.array_equal(tm, otm)


@pytest.mark.parametrize("kind", ("long", "dense", "both"))
def test_fp32_rows_keep_their_photons(kind):
    from crvgpu import lookup as LK
    L, rows = _rows(kind)
    eng, D = LK.SubstepEngine(), LK.DeviceLookup(L)
    s, c, t = (x.cpu().numpy() for x in eng.run(D, LK.DeviceRows(rows), 9, precision="fp32"))
    if kind == "long":
        want = len(O.substep_photons(L, rows, 9)[0])
        assert abs(len(s) - want) < 6 * np.sqrt(want) + 0.01 * want  # (Poisson, and the draws' 24-bit uniforms)
    for r in (0, 1, 2, 5, 40, 47, 119):
        one = {k: v[r:r + 1] for k, v in rows.items()}
        s1, c1, t1 = (x.cpu().numpy() for x in eng.run(D, LK.DeviceRows(one), 9, precision="fp32"))
        m = (s == rows["step"][r]) & (c == rows["chan"][r])
        assert np.array_equal(t[m], t1)


@pytest.mark.parametrize("columns", (2, 5, 129))
def test_emissions_dealt_out_equal_the_oracle(columns):
    """FP64 fibre decay with at most 1, 4 and 128 emissions per arrival (more blocks than are dealt out at a time)."""
    import copy

    from crvgpu import lookup as LK
    L, rows = _rows("long")
    L, rng = copy.deepcopy(L), np.random.default_rng(columns)
    L.fiber_decay_time = 7.4
    for t in L.tables.values():
        t.emis = rng.integers(0, 3, (len(t.prob), columns)).astype(np.uint8)
        t.emis[:, -1] += 1
        t.emis_sum = t.emis.sum(1, dtype=np.int32)
    st, ch, tm = LK.substep_photons(L, rows, 4)
    ost, och, otm, lim = O.substep_photons(L, rows, 4)
    assert not lim and len(st) > 1000
    assert np.array_equal(st, ost) and np.array_equal(ch, och) and np.array_equal(tm, otm)
