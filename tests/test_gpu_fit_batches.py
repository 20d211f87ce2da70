"""The fit of a batch in one launch against the launches by rounds, in which every lane works for itself: batches from one
waveform per warp to several per lane, waveforms on both sides of the lengths that the warp copies and searches together,
windows on both sides of the points that the FP64 evaluation deals out, more points than it deals out at a time.  Same
operations in the same order: exact."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _batch(n, seed):
    """Pulses of 20 to 2,000 ADC on waveforms of 1 to 300 samples, one in four cut off flat (plateaus of up to 60 samples)."""
    r = np.random.default_rng(seed)
    lens = r.choice([1, 2, 12, 31, 32, 33, 34, 47, 48, 49, 63, 64, 65, 66, 97, 300], n)
    off = np.cumsum(lens) - lens
    wf = np.repeat(np.arange(n), lens)
    pos = np.arange(int(lens.sum())) - off[wf]
    y = 100.0 + 2.0 * r.standard_normal(len(pos))
    for k in range(5):
        beta, mu = r.uniform(3, 45, n), r.uniform(-0.1, 1.05, n) * lens
        amp = np.where(r.integers(0, 6, n) > k, np.exp(r.uniform(np.log(60), np.log(6000), n)), 0.0)
        z = (pos - mu[wf]) * 12.55 / beta[wf]
        y += amp[wf] * np.exp(-z - np.exp(-np.clip(z, -50, None)))
    flat = (r.random(n) < 0.25)[wf]
    y = np.where(flat, np.minimum(y, 130.0), y)
    y = np.where(flat, np.round(y / 30.0) * 30.0, y)
    return off, lens, r.integers(-100, 500, n), np.clip(np.round(y), 0, 4095).astype(np.int16)


@pytest.mark.parametrize("precision", ("fp32", "fp64"))
@pytest.mark.parametrize("n", (1, 33, 700, 2500, 12001))
def test_one_launch_equals_the_rounds(n, precision):
    import torch
    from crvgpu import config as CF
    from crvgpu import pulsefit as PF
    from crvgpu.params import make_params
    off, lens, start, adc = _batch(n, 5 + n)
    P = make_params(reco=CF.RecoConfig(), precision=precision)
    P.period = 12.55
    up = lambda a, t: torch.from_numpy(np.ascontiguousarray(np.asarray(a, t))).cuda()  # noqa: E731
    one = np.ones(n)
    out = []
    try:
        for shape in (PF.DEFAULT_SHAPE, (128, 16, 3)):
            PF.set_shape(shape)
            eng = PF.PulseEngine()
            eng.out_factor = 16.0
            r = eng.run(P, up(off, np.int64), up(lens, np.int32), up(start, np.int64), up(100 * one, float),
                        up(400 * one, float), up(27 * one, float), adc16=up(adc, np.int16), max_pulses=2 ** 31 - 1,
                        nsamples=len(adc))
            out.append({k: v.cpu().numpy() for k, v in r.items()})
    finally:
        PF.set_shape(PF.DEFAULT_SHAPE)
    a, b = out
    assert n < 700 or len(a["pe"]) > n
    for k in b:
        assert np.array_equal(a[k], b[k], equal_nan=a[k].dtype.kind == "f"), k
