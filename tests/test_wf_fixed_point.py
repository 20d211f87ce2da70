"""FP64 synthesis: first samples and template indices decided on fixed-point copies, against the FP64 forms they stand for."""
import numpy as np

f32 = np.float32


def d2fx(x):
    return int(np.trunc(np.float64(x) * 2.0 ** 32))       # exact product, truncated


def test_certain_decisions_equal_the_fp64_forms():
    rng = np.random.default_rng(6)
    certain = 0
    for P, prec, reach in ((12.55, 0.5, 100.0), (12.5, 0.25, 60.0), (7.3, 0.1, 30.0)):
        Pfx, unit = d2fx(P), f32(2.0 ** -20 / prec)
        top = reach + 3 * P
        half = f32(0.5) - f32(4.0) * (f32(top / prec) * f32(2.0 ** -22) + f32(16.0) * unit)
        for _ in range(4000):
            ts = float(rng.uniform(-50, 1e5))
            j = int(rng.integers(0, 300))
            st_want = rng.choice([rng.uniform(-1, top), rng.integers(0, 200) * prec + prec / 2 + rng.normal(0, 1e-5),
                                  rng.normal(0, 1e-5), rng.integers(0, 5) * P + rng.normal(0, 1e-9)])
            t = float(j * P + ts - st_want)
            x = d2fx(t - ts)
            # first sample
            exact = max(0, int(np.ceil((t - ts) / P)))
            if x <= -16:
                assert exact == 0
            elif x >= 16:
                k = x // Pfx
                r, tol = x - k * Pfx, k + 8
                if not (r < tol or Pfx - r < tol):
                    assert k + 1 == exact, (t, ts)
                    certain += 1
            # template index: the pair's time, positive and up to the reach
            st = float(j) * P + ts - t
            if st > top:
                continue
            d = ((j * Pfx) >> 12) - (x >> 12)
            d = (d + 2 ** 31) % 2 ** 32 - 2 ** 31
            xq = f32(f32(d) * unit)
            r = np.rint(xq)
            if d < -16:
                assert st < 0
            elif d >= 16 and abs(f32(xq - r)) <= half:
                assert st >= 0 and int(r) == int(np.rint(st / prec)), (st, d)
                certain += 1
    assert certain > 10000
