"""Crossings whose parameter rounds to zero, of either sign, on an edge with others: both
zeros are one parameter, so the later other edge comes first whatever form orders the edge's
insertions (a thread to 8, a warp to 256, a block beyond), against the oracle (bit for bit)."""
from fractions import Fraction

import numpy as np
import pytest

import pyoracle
from gcmfgh import synth

START, END = np.array([1.0 / 3.0, 1.0 / 7.0]), np.array([4001.1, 0.2])


def _area(a, b, c):
    return (b[0] - a[0]) * (c[1] - a[1]) - (b[1] - a[1]) * (c[0] - a[0])


def _sign(a, b, c):
    a, b, c = ([Fraction(float(x)) for x in v] for v in (a, b, c))
    d = (b[0] - a[0]) * (c[1] - a[1]) - (b[1] - a[1]) * (c[0] - a[0])
    return (d > 0) - (d < 0)


def _spike(rng, down):
    """(foot, tip, foot): a spike of no visible width through START, down or up to its tip.  Both its
    edges leave START strictly on END's other side, by less than START's area can show."""
    while True:
        tip = START + rng.uniform([-0.05, 0.3], [0.05, 0.4]) * (-1.0 if down else 1.0)
        feet = []
        for _ in range(400):
            f = START - rng.uniform(0.5, 2.0) * (tip - START) + rng.integers(-2, 3, 2) * 2.0 ** -54
            if _area(START, f, tip) == 0.0 and _sign(START, f, tip) * _sign(END, f, tip) < 0:
                feet.append(f)
            if len(feet) == 2:
                return feet[0], tip, feet[1]


def _pair(count, seed):
    """A strip from START to END, and a comb that crosses the strip's first edge `count` times, the
    spike's two crossings among them.  The strip is the longer ring for odd seeds, the spike
    points down (and its foot's way out is one more crossing) from seed 2 on."""
    rng = np.random.default_rng(seed)
    down = seed >= 2
    left = count - 3 if down else count - 2
    teeth = left // 2
    comb = list(_spike(rng, down))
    for i in range(teeth):
        x = 3.0 + 3.0 * i
        comb += [np.array(v) for v in ((x, -1.0), (x + 0.5, 0.5), (x + 1.0, -1.0))]
    end = 3.0 * teeth + 4.0
    comb += [np.array([end, -1.0])]
    if left % 2:                                    # the last crossing: into the strip and out over its far side
        comb += [np.array([end + 0.25, 3.0]), np.array([5000.0, 3.0])]
    comb += [np.array([5000.0, -3.0]), np.array([-3.0, -3.0])]
    far = np.linspace(4001.0, -2.0, 3 * count + 20 if seed % 2 else 2)
    strip = [START, END] + [np.array([x, 1.0 + 0.01 * (i % 2)]) for i, x in enumerate(far)]
    return np.array(strip), np.array(comb)


def _crossings_of_first_edge(P, Q):
    """How many, and for those with a parameter of zero the sign bits, in Q's order."""
    n = 0
    zeros = []
    for i in range(len(Q)):
        a, b = Q[i], Q[(i + 1) % len(Q)]
        if _sign(START, a, b) * _sign(END, a, b) < 0 and _sign(a, START, END) * _sign(b, START, END) < 0:
            n += 1
            t = _area(START, a, b) / (_area(START, a, b) - _area(END, a, b))
            if t == 0.0:
                zeros.append(bool(np.signbit(t)))
    return n, zeros


COUNTS = [4, 7, 8, 9, 10, 31, 32, 33, 65, 255, 256, 257, 513, 700]


@pytest.mark.parametrize("count", COUNTS)
def test_inputs(count):
    """The crossings are as many as the case says, and both zeros are among their parameters, each
    first in some pair."""
    for seed in range(4):
        n, zeros = _crossings_of_first_edge(*_pair(count, seed))
        assert n == count and zeros == ([True, False] if seed >= 2 else [False, True])


@pytest.mark.gpu
@pytest.mark.parametrize("count", COUNTS)
def test_order_at_zero(engine, count):
    import gcmfgh
    pairs = [_pair(count, seed) for seed in range(4)]
    strips, combs = [p for p, _ in pairs], [q for _, q in pairs]
    base, ovl = synth.Layer.from_rings(strips + combs), synth.Layer.from_rings(combs + strips)
    ids = np.arange(8, dtype=np.int32)
    try:
        engine.set_precision(True)
        for union in (False, True):
            engine.set_params(1e-7, 0.0, union)
            engine.clip_batch(gcmfgh.DeviceLayer(base), gcmfgh.DeviceLayer(ovl), ids, ids)
            r = engine.clip_result()
            o = pyoracle.clip_batch(base, ovl, ids, ids, eps_clean=0.0, union=union, exact=True)
            assert np.array_equal(r.status, o.status)
            assert np.array_equal(r.comp_size, o.comp_size)
            assert np.array_equal(r.xy, o.xy)
    finally:
        engine.set_precision(False)
        engine.set_params(1e-7, 1e-7, False)
