"""GPU coincidence finder against the oracle at the edges of its passes: events around the shared-memory pass's 192 hits,
several sector types, more than 32 hits within one link window.  Membership identical; properties within 1e-12 relative
(sums of at most a few hundred FP64 terms in another order)."""
from dataclasses import replace

import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("modules,hits,span", [(1, (1, 2, 33, 191, 192, 193, 260), 1500.0), (1, (64, 192, 200), 25.0),
                                               (6, (40, 300), 400.0)])
def test_event_sizes_match_the_oracle(modules, hits, span):
    from crvgpu import coinc as CO
    from crvgpu import config as CF
    from crvgpu import geometry as GM
    rng = np.random.default_rng(modules + int(span))
    geom = GM.module_geometry(modules)
    G = GM.sector_geom(geom)
    base = replace(CF.WORKLOAD_CUTS)
    cfg = CF.FinderConfig(cuts={n: base if i % 2 == 0 else replace(base, max_dt=14.0, coincidence_layers=2, pe_threshold=5.0)
                                for i, n in enumerate(G.sector_names)})
    status = np.zeros(4 * geom.nbars, np.int64)
    n = sum(hits)
    ev = np.repeat(np.arange(len(hits)), hits)
    tracks = rng.uniform(0, span, (len(hits), 6))
    on = rng.random(n) < 0.6                              # hits of tracks: neighbouring counters near one time
    col, mod = rng.integers(4, 8, n), rng.integers(0, modules, n)
    bar = np.where(on, mod * 64 + rng.integers(0, 4, n) * 16 + col, rng.integers(0, geom.nbars, n))
    t = np.where(on, tracks[ev, rng.integers(0, 6, n)] + rng.normal(0, 3, n), rng.uniform(0, span, n))
    pe, sipm, seq = rng.exponential(20, n), rng.integers(0, 4, n), np.zeros(n, np.int64)
    idx = np.arange(n) - np.repeat(np.cumsum(hits) - np.array(hits), hits)
    cl, mem = CO.find_events(ev, idx, bar, sipm, t, pe, seq, G, status, cfg)
    rows = CO.rows_of(cl, mem)
    at = 0
    for e in range(len(hits)):
        m = ev == e
        want = O.find_event({"idx": idx[m], "bar": bar[m], "sipm": sipm[m], "time": t[m], "pe": pe[m], "seq": seq[m]}, G,
                            status, cfg)
        got = [r for r, k in zip(rows, cl["event"]) if k == e]
        assert len(got) == len(want), (e, hits[e])
        for r, w in zip(got, want):
            assert [int(v) for v in r["pulses"]] == [int(v) for v in w["pulses"]], (e, hits[e])
            for k in ("pe", "start", "end", "slope", "avgtime"):
                np.testing.assert_allclose(r[k], w[k], rtol=1e-12, atol=1e-9)
        at += len(want)
    assert at == len(rows) > 0
