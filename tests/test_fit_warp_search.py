"""The warp's part of the peak search reads samples that one lane wrote (a copy, or the samples less its pulse): a warp
barrier orders them, which votes and shuffles do not."""
import os
import re

import numpy as np
import pytest

SRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "mu2e-fastsim_gb300", "csrc",
                   "crv_pulsefit.cuh")


def test_a_barrier_comes_before_the_search():
    """No result shows a missing barrier for certain, so the source is read: every lane passes one on entry, ahead of the
    first sample that the search reads and of anything that could leave a lane out."""
    text = re.sub(r"//[^\n]*", "", open(SRC).read())
    body = text[text.index("bool pf_search_warp("):]
    body = body[body.index("{"):body.index("\n}\n")]
    at = body.index("__syncwarp();")
    assert at < body.index("peak_scan<R>") < body.index("peak_scan_warp<R>")
    assert not re.search(r"\b(if|while|for|return)\b", body[:at])


@pytest.mark.gpu
@pytest.mark.parametrize("precision", ("fp32", "fp64"))
def test_pulses_far_apart_equal_the_rounds(precision):
    """Every pulse is followed by more samples than a lane searches alone (32), so each search after a subtraction is the
    warp's; against the launches by rounds, where each lane searches its own samples: exact, three times."""
    import torch
    from crvgpu import config as CF
    from crvgpu import pulsefit as PF
    from crvgpu.params import make_params
    r = np.random.default_rng(11)
    n, L = 3000, 256
    lens = r.integers(200, L + 1, n)
    pos = np.arange(L)[None, :]
    y = 100.0 + 2.0 * r.standard_normal((n, L))
    for k in range(5):
        z = (pos - (15 + 48 * k + r.uniform(-3, 3, (n, 1)))) * 12.55 / r.uniform(10, 25, (n, 1))
        y += r.uniform(100, 2000, (n, 1)) * np.exp(-z - np.exp(-np.clip(z, -50, None)))
    adc = np.concatenate([np.clip(np.round(v[:m]), 0, 4095) for v, m in zip(y, lens)]).astype(np.int16)
    P = make_params(reco=CF.RecoConfig(), precision=precision)
    P.period = 12.55
    up = lambda a, t: torch.from_numpy(np.ascontiguousarray(np.asarray(a, t))).cuda()  # noqa: E731
    one, out = np.ones(n), []
    try:
        for shape in ((128, 16, 3),) + 3 * (PF.DEFAULT_SHAPE,):
            PF.set_shape(shape)
            eng = PF.PulseEngine()
            eng.out_factor = 16.0
            a = eng.run(P, up(np.cumsum(lens) - lens, np.int64), up(lens, np.int32), up(0 * one, np.int64),
                        up(100 * one, float), up(400 * one, float), up(27 * one, float), adc16=up(adc, np.int16),
                        max_pulses=2 ** 31 - 1, nsamples=len(adc))
            out.append({k: v.cpu().numpy() for k, v in a.items()})
    finally:
        PF.set_shape(PF.DEFAULT_SHAPE)
    assert len(out[0]["pe"]) > 3 * n
    for b in out[1:]:
        for k in b:
            assert np.array_equal(out[0][k], b[k], equal_nan=b[k].dtype.kind == "f"), k
