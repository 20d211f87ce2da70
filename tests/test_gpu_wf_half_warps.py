"""FP32-mixed synthesis of many SiPMs, two per warp, against the same SiPMs in batches small enough for a warp each: clusters
of 8 to 20 samples (16 is the most that half a warp takes), more charges than are staged at a time, several clusters per
SiPM, odd numbers of SiPMs, with and without noise.  Same operations in the same order: exact."""
from dataclasses import replace

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,mean,span,noise", [(20001, 12, 15.0, True), (16000, 25, 90.0, True), (9973, 25, 110.0, False),
                                               (6007, 300, 60.0, True)])
def test_batches_of_any_size_give_the_same_digis(n, mean, span, noise):
    from crvgpu import chain as CH
    from crvgpu import config as CF
    from crvgpu import geometry as GM
    geom = GM.module_geometry(1)
    cond = GM.default_conditions(geom)
    rng = np.random.default_rng(n)
    nc = 4 * geom.nbars
    lab = (np.arange(n) // 150 + 1) * 32768 + np.sort(rng.permuted(np.tile(np.arange(nc), (n // 150 + 1, 1)), axis=1)[:, :150],
                                                     axis=1).ravel()[:n]
    k = 1 + rng.poisson(mean, n)
    label = np.repeat(lab, k)
    burst = np.where(rng.random(len(label)) < 0.2, 400.0, 0.0)
    t = np.repeat(rng.uniform(20, 900, n), k) + burst + rng.uniform(0, np.repeat(rng.uniform(1, span, n), k))
    o = np.lexsort((t, label))
    Q = {"chan": label[o], "time": t[o], "charge": 2.652e-13 * rng.uniform(0.3, 2.0, len(o))}
    cfg = CF.ChainConfig(precision="fp32")
    cfg = replace(cfg, noise=noise)
    whole = CH.digis(Q, cond, cfg, None, key=11, geom=geom)
    assert len(whole["chan"]) > n // 2
    parts, cut = [], np.searchsorted(Q["chan"], lab[::1500])
    for a, b in zip(cut, np.append(cut[1:], len(o))):
        parts.append(CH.digis({c: v[a:b] for c, v in Q.items()}, cond, cfg, None, key=11, geom=geom))
    for c in whole:
        assert np.array_equal(whole[c], np.concatenate([p[c] for p in parts])), c
