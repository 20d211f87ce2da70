"""Large events whose earlier sector types give a cluster of one member for every hit (cuts of one layer, no combination check):
the later types' records then lie where they were found and only their members' places change.  Against the oracle:
membership identical, properties within 1e-12 relative (sums of a few FP64 terms)."""
from dataclasses import replace

import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _event(geom, G, singles, pairs, rng):
    """Hits 100 ns apart: alone in the types of `singles`, two SiPMs of one side together in those of `pairs`."""
    bar, sipm, t = [], [], []
    for ty in np.unique(G.sector_type[G.sector]):
        bars = np.flatnonzero(G.sector_type[G.sector] == ty)
        for k in range(90 if ty in singles or ty in pairs else 0):
            b, at = int(rng.choice(bars)), 100.0 * (len(t) + 1)
            for s in ((0,) if ty in singles else (0, 2)):
                bar.append(b)
                sipm.append(s)
                t.append(at + s)
    o = rng.permutation(len(t))
    return {"bar": np.array(bar)[o], "sipm": np.array(sipm)[o], "time": np.array(t)[o], "idx": np.arange(len(t)),
            "pe": rng.uniform(20, 90, len(t)), "seq": np.zeros(len(t), np.int64)}


@pytest.mark.parametrize("order", ("singles first", "singles last", "all singles", "gap"))
def test_single_member_clusters_of_large_events(order):
    from crvgpu import coinc as CO
    from crvgpu import config as CF
    from crvgpu import geometry as GM
    rng = np.random.default_rng(8)
    geom = GM.module_geometry(12)
    G = GM.sector_geom(geom)
    types = [int(v) for v in np.unique(G.sector_type[G.sector])]
    assert len(types) >= 4
    singles, pairs = {"singles first": (types[:2], types[2:]), "singles last": (types[-1:], types[:-1]),
                      "all singles": (types, []), "gap": (types[1:2], types[3:])}[order]
    cuts = replace(CF.WORKLOAD_CUTS, coincidence_layers=1, pe_threshold=1.0)
    cfg = CF.FinderConfig(cuts={n: cuts for n in G.sector_names}, big_cluster_threshold=0)
    status = np.zeros(4 * geom.nbars, np.int64)
    ev = _event(geom, G, singles, pairs, rng)
    assert len(ev["bar"]) > 192                           # (more hits than the shared-memory pass takes)
    rows, want = CO.find_event(ev, G, status, cfg), O.find_event(ev, G, status, cfg)
    assert len(rows) == len(want) >= 180
    assert sum(len(w["pulses"]) == 1 for w in want) >= 90
    for r, w in zip(rows, want):
        assert [int(v) for v in r["pulses"]] == [int(v) for v in w["pulses"]]
        for k in ("pe", "start", "end", "avgtime"):          # (no slope: one layer)
            np.testing.assert_allclose(r[k], w[k], rtol=1e-12, atol=1e-9)
