"""FP64 lookup photons with arrival probabilities that are not numbers, above 1, infinite or negative (a channel's deviation, a
table entry): the oracle's photons, bit for bit (a probability that is not below 1 counts as 1)."""
import copy

import numpy as np
import pytest

from oracle import oracle as O
from tests.test_oracle_lookup import lookup_fixture

pytestmark = pytest.mark.gpu
ODD = (np.nan, -np.nan, np.inf, -np.inf, 1e38, -1.0)


@pytest.mark.parametrize("where", ("deviation", "table", "both"))
@pytest.mark.parametrize("mu", (False, True))
def test_odd_probabilities_equal_the_oracle(where, mu):
    from crvgpu import lookup as LK
    L, rows, _ = lookup_fixture()
    L, rows = copy.deepcopy(L), {k: np.array(v)[:400] for k, v in rows.items() if mu or k != "mu"}
    for k in ("n_scint", "n_ck_s", "n_ck_f"):
        rows[k] = np.minimum(rows[k], 20)
    if where != "table":
        rows["dev"][::5] = np.resize(ODD, len(rows["dev"][::5]))
    if where != "deviation":
        for t in L.tables.values():
            t.prob = np.array(t.prob)
            t.prob[::3] = np.resize(np.asarray(ODD, np.float32), len(t.prob[::3]))
    st, ch, tm = LK.substep_photons(L, rows, 13)
    ost, och, otm, lim = O.substep_photons(L, rows, 13)
    assert not lim and len(st) > 1000
    if where == "deviation":             # rows whose deviation is not a number have photons (a step of their own each)
        assert np.isin(rows["step"][np.isnan(rows["dev"]) & (rows["nsub"] > 100)], ost).any()
    assert np.array_equal(st, ost) and np.array_equal(ch, och) and np.array_equal(tm, otm)
