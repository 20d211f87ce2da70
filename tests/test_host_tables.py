"""Host tables of the drop-in calls: recycled memory, modules and waveform matrices built without loops, and synthesize's
cluster marks from the device against those from the host.  Exact."""
import gc
import threading

import numpy as np
import pytest


def test_recycled_memory_is_never_shared_and_bounded():
    from crvgpu.hostmem import SMALL, HostPool
    pool = HostPool(limit=8 * SMALL)
    a = pool.empty((3, SMALL // 8), np.float64)
    a[:] = 7.0
    view, at = a[1:, 5:], a.__array_interface__["data"][0]
    del a
    b = pool.empty((3, SMALL // 8), np.float64)
    b[:] = 1.0
    assert (view == 7.0).all() and not np.shares_memory(view, b)          # a view keeps the block
    del view
    gc.collect()
    c = pool.empty(3 * SMALL // 4, np.int32)                              # same size class: the first block again
    assert c.__array_interface__["data"][0] == at and c.flags.writeable and pool.kept == 0
    small = pool.empty(10, np.int16)
    assert small.base is None and small.dtype == np.int16
    del b, c
    blocks = [pool.empty(3 * SMALL, np.uint8) for _ in range(6)]
    big = pool.empty(9 * SMALL, np.uint8)
    del blocks, big
    gc.collect()
    assert 0 < pool.kept <= 8 * SMALL
    pool.release()
    assert pool.kept == 0 and not pool._free


@pytest.mark.parametrize("n", (1, 1 << 20, (1 << 20) + 1, 33554432, 32190432, 10 ** 9 + 7))
def test_size_classes(n):
    from crvgpu.hostmem import HostPool
    c = HostPool.size_class(n)
    assert n <= c <= n + n // 8 + 1 and HostPool.size_class(c) == c


def test_threads_never_hold_the_same_block():
    from crvgpu.hostmem import SMALL, HostPool
    pool, bad = HostPool(), []

    def work(k):
        for i in range(200):
            a = pool.empty(SMALL, np.uint8)
            a[::4096] = k
            b = pool.empty(SMALL, np.uint8)
            b[::4096] = 100 + k
            if not ((a[::4096] == k).all() and (b[::4096] == 100 + k).all()):
                bad.append(k)
            del a, b

    ts = [threading.Thread(target=work, args=(k,)) for k in range(8)]
    [t.start() for t in ts]
    [t.join() for t in ts]
    assert not bad


@pytest.mark.parametrize("n,lengths,layers,counters", [(1, None, 4, 16), (7, None, 4, 16), (3, [4500.0, 2300.0, 4500], 2, 5),
                                                       (0, None, 4, 16)])
def test_module_geometry(n, lengths, layers, counters):
    from crvgpu import geometry as G
    g = G.module_geometry(n, lengths, n_layers=layers, n_counters=counters)
    ls = lengths if lengths is not None else \
        [4500.0] if n == 1 else list(np.random.default_rng(0).choice(G.LENGTHS, n))
    seen, order, i = {}, sorted(set(float(v) for v in ls)), 0
    for m, length in enumerate(ls):
        s = 0 if n == 1 else order.index(float(length))
        seen[s] = seen.get(s, -1) + 1
        for layer in range(layers):
            for c in range(counters):
                x = m * (counters * G.PITCH + G.MODULE_GAP) + (c - (counters - 1) / 2) * G.PITCH + G.STAGGER * (layer % 2)
                assert (g.sector[i], g.module[i], g.layer[i], g.counter[i]) == (s, seen[s], layer, c)
                assert tuple(g.center[i]) == (x, (layer - (layers - 1) / 2) * G.LAYER_PITCH, 0.0)
                assert tuple(g.halflen[i]) == (G.WIDTH / 2, G.THICK / 2, float(length) / 2)
                i += 1
    assert g.nbars == i


@pytest.mark.parametrize("dt", (np.int16, np.int64))
@pytest.mark.parametrize("runs", ([1], [2, 1, 3], [1] * 9, [4, 1, 1, 2, 1, 1, 4], [1, 5]))
def test_waveform_matrix(runs, dt):
    from crvgpu.pulsefit import concat_waveforms
    rng = np.random.default_rng(len(runs))
    L, nd = 12, sum(runs)
    bar = np.repeat(np.arange(len(runs)), runs)
    start = np.concatenate([100 + L * np.arange(r) for r in runs])
    adc = rng.integers(-4096, 4096, (nd, L)).astype(dt)
    gid, mat, n, st, first = concat_waveforms(bar * 0, bar, bar * 0, start, adc.ravel(), np.full(nd, L))
    want, at = np.zeros((len(runs), max(runs) * L), np.int64), 0
    for i, r in enumerate(runs):
        want[i, :r * L] = adc[at:at + r].ravel()
        at += r
    assert mat.dtype == np.int64 and np.array_equal(mat, want) and np.array_equal(gid, bar)
    assert np.array_equal(n, np.array(runs) * L) and np.array_equal(st, start[first])


def test_waveform_matrix_stays_in_its_arrays():
    from crvgpu import _capi
    adc, mat = np.zeros((4, 3), np.int16), np.full((2, 6), 9, np.int64)
    f = lambda a: np.asarray(a, np.int64)  # noqa: E731
    p = lambda a: a.ctypes.data  # noqa: E731
    for first, ndig in (([0, 3], [1, 2]), ([-1, 0], [1, 1]), ([0, 1], [1, 3]), ([0, 1], [1, -1])):
        a, b = f(first), f(ndig)
        assert _capi.load().crv_waveform_matrix(2, 2, 3, p(a), p(b), p(adc), 4, p(mat)) == _capi.CRV_ERR_ARG
        assert (mat[1] == 9).all()


@pytest.mark.gpu
@pytest.mark.parametrize("order", ("sorted", "grouped"))
@pytest.mark.parametrize("cut", (10 ** 6, 40, 1))
def test_synthesize_takes_labels_of_any_type(order, cut):
    """Labels that the device compares (int64, int32) and labels that the host compares (float64), with the caller's TDC0
    evaluated batch by batch."""
    from crvgpu import waveform as WF
    rng = np.random.default_rng(3)
    lab = np.repeat(rng.permutation(40) if order == "grouped" else np.arange(40), 5)
    time = np.concatenate([np.sort(rng.uniform(0, 900, 5)) for _ in range(40)])
    charge = rng.uniform(0.5, 30.0, 200) * 2.652e-13

    def run(dt):
        asked = []

        def tdc0(c):
            asked.append(np.asarray(c, np.int64).tolist())
            return 0.1 * np.asarray(c, float)

        return WF.synthesize(lab.astype(dt), time, charge, tdc0, max_charges=cut), asked

    want, asked = run(np.float64)
    assert len(want["chan"]) and (len(asked) > 1) == (cut < 200)
    for dt in (np.int64, np.int32):
        got, seen = run(dt)
        assert seen == asked
        assert all(np.array_equal(got[k], want[k]) for k in want)
    with pytest.raises(ValueError, match="grouped"):
        WF.synthesize(np.array([3, 1, 3]), np.arange(3.0), np.ones(3), lambda c: 0.0 * np.asarray(c, float))
    with pytest.raises(ValueError, match="non-negative"):
        WF.synthesize(np.array([-3, 1]), np.arange(2.0), np.ones(2), lambda c: 0.0 * np.asarray(c, float))
