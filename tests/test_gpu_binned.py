"""Binned pairs' one-pass count + emit: every pair's edges through the grid, its listing
classes and the FP32 tests, against the oracle -- degenerate lattice pairs, edges far longer
than the grid (outside the FP32 copies' range), common boxes of no width, tiny and remote
coordinates, and a record count beyond the first capacity."""
import numpy as np
import pytest

import pyoracle
from gcmfgh import synth

pytestmark = pytest.mark.gpu


def _pairs():
    rng = np.random.default_rng(77)
    pairs = synth.degeneracy_pairs(77, 120, 4, 300)[1]
    for k in range(200):
        q = 0.5 ** rng.integers(0, 3)
        pairs.append(tuple(np.round(synth._star(rng, int(rng.integers(4, 50)), 0.0, 0.0, 6.0, 0.2, 1.0) / q) * q
                           for _ in range(2)))
    for scale, shift in ((1e-9, 0.0), (1e9, 0.0), (1.0, 1e8), (1e-3, 1e3)):
        for n, m in ((3, 400), (33, 31), (257, 1)):
            P = synth._star(rng, n, 0.0, 0.0, 1.0, 0.5, 1.0) * scale + shift
            Q = synth._star(rng, max(m, 3), 0.1, 0.1, 1.0, 0.5, 1.0) * scale + shift
            pairs.append((P, Q))
    # long edges across a small polygon, and boxes that touch in one line
    for n in (8, 200):
        P = synth._star(rng, n, 0.0, 0.0, 1.0, 0.5, 1.0)
        pairs.append((P, np.array([[-5e6, -0.1], [5e6, 0.0], [5e6, 0.1], [-5e6, 0.2]])))
        x = P[:, 0].max()
        pairs.append((P, np.array([[x, -1.0], [x + 1.0, -1.0], [x + 1.0, 1.0], [x, 1.0]])))
    return pairs


@pytest.mark.parametrize("exact", [False, True])
@pytest.mark.parametrize("hint", [0, 1])
def test_every_pair_binned(engine, exact, hint):
    import gcmfgh
    pairs = _pairs()
    base, ovl = (synth.Layer.from_rings([p[i] for p in pairs]) for i in (0, 1))
    ids = np.arange(len(pairs), dtype=np.int32)
    db, do = gcmfgh.DeviceLayer(base), gcmfgh.DeviceLayer(ovl)
    try:
        engine.set_tuning(bin_grid=0, record_hint=hint)      # 1: the arrays are short, the pass runs again
        engine.set_precision(exact)
        engine.clip_batch(db, do, ids, ids)
        r = engine.clip_result()
    finally:
        engine.set_tuning(bin_grid=1 << 16, record_hint=0)
        engine.set_precision(False)
    o = pyoracle.clip_batch(base, ovl, ids, ids, exact=exact)
    assert np.array_equal(r.status, o.status)
    assert np.array_equal(r.count1[r.status != 2], o.count1[o.status != 2])
    assert np.array_equal(r.ncomp, o.ncomp)
    assert np.array_equal(r.comp_size, o.comp_size)
    assert np.array_equal(r.xy, o.xy)


def _near_pairs(exponent):
    """Pairs whose vertices lie close to the other ring's edges, at sizes whose products
    underflow, overflow or just fit FP32."""
    rng = np.random.default_rng(12)
    pairs = []
    for n in [3, 4, 5, 8, 17, 40] * 50:
        P = synth._star(rng, n, 0.0, 0.0, 1.0, 0.5, 1.0)
        Q = P * (1.0 + rng.choice([1e-1, 1e-2, 1e-8]) * rng.uniform(-1.0, 1.0, size=P.shape))
        pairs.append((P * 2.0 ** exponent, np.roll(Q * 2.0 ** exponent, 1, 0)))
    return pairs


def _underflow_pairs(exponent):
    """Pairs with an edge that ends 2^-26 beyond another: of 400,000, those that a side test on
    FP32 copies whose margins underflow would take to be apart."""
    rng = np.random.default_rng(1)
    n, s = 400_000, 2.0 ** exponent
    p1, p2 = rng.uniform(0.0, 1.0, (n, 2)), rng.uniform(0.0, 1.0, (n, 2))
    d = p2 - p1
    normal = np.stack([-d[:, 1], d[:, 0]], 1)
    at = p1 + rng.uniform(0.1, 0.9, (n, 1)) * d
    q1 = at + normal * rng.uniform(0.1, 1.2, (n, 1)) * 2.0 ** -26
    q2 = at - normal * rng.uniform(0.3, 1.0, (n, 1))
    f1, f2, g1, g2 = ((v * s).astype(np.float32) for v in (p1, p2, q1, q2))
    M = np.float32(2.0 * s)
    e, a, b = f2 - f1, g1 - f1, g2 - f1
    norm = lambda v: np.abs(v[:, 0]) + np.abs(v[:, 1])                     # noqa: E731
    with np.errstate(under="ignore"):
        s1, s2 = (e[:, 0] * v[:, 1] - e[:, 1] * v[:, 0] for v in (a, b))
        m1, m2 = (M * np.float32(2.0 ** -19) * (norm(e) + M * np.float32(2.0 ** -24) + norm(v)) for v in (a, b))
    apart = ((s1 > m1) & (s2 > m2)) | ((s1 < -m1) & (s2 < -m2))
    inside = (np.minimum(q1, q2) > 0.0).all(1) & (np.maximum(q1, q2) < 1.0).all(1)
    # (the far corners make the common box the unit square)
    return [(np.array([p1[i], p2[i], [1.0, 1.0], [0.0, 0.0]]) * s, np.array([q1[i], q2[i], [1.0, 0.0], [0.0, 1.0]]) * s)
            for i in np.nonzero(apart & inside)[0]]


@pytest.mark.parametrize("exponent", [-90, -68, -67, -66, -52, -51, -50, -48, 56, 58, 60, 62, 64, 100])
def test_sizes_beyond_fp32(engine, exponent):
    import gcmfgh
    pairs = _near_pairs(exponent)
    if -68 <= exponent <= -66:
        beyond = _underflow_pairs(exponent)
        assert len(beyond) >= 3
        pairs += beyond
    base, ovl = (synth.Layer.from_rings([p[i] for p in pairs]) for i in (0, 1))
    ids = np.arange(len(pairs), dtype=np.int32)
    try:
        engine.set_tuning(bin_grid=0)
        engine.set_precision(True)
        engine.set_params(1e-7, 0.0, False)
        engine.clip_batch(gcmfgh.DeviceLayer(base), gcmfgh.DeviceLayer(ovl), ids, ids)
        r = engine.clip_result()
    finally:
        engine.set_tuning(bin_grid=1 << 16)
        engine.set_precision(False)
        engine.set_params(1e-7, 1e-7, False)
    o = pyoracle.clip_batch(base, ovl, ids, ids, eps_clean=0.0, exact=True)
    assert np.array_equal(r.status, o.status)
    assert np.array_equal(r.count1[r.status != 2], o.count1[o.status != 2])
    assert np.array_equal(r.comp_size, o.comp_size)
    assert np.array_equal(r.xy, o.xy)


def test_more_listings_than_copies(engine):
    """Two rings of a million edges, some of one right across it: about 9e8 listings, beyond
    what FP32 copies are made for.  Against the two passes, which make none (and which smaller
    pairs are compared with the oracle for)."""
    import gcmfgh
    n, longs = 1_000_000, 1500
    rng = np.random.default_rng(8)
    a = np.linspace(0.0, 2.0 * np.pi, n, endpoint=False)
    r = 1.0 + 1e-4 * rng.uniform(-1.0, 1.0, n)
    r[np.arange(longs) * (n // longs)] = -1.0                   # a spike to the far side and back
    Q = np.stack([r * np.cos(a), r * np.sin(a)], 1)
    b = np.linspace(0.0, 2.0 * np.pi, n + 100, endpoint=False)
    s = 1.0002 * (1.0 - 0.5 * np.exp(-((b - 1.0) / 0.3) ** 2))  # dented, else around the other
    P = np.stack([s * np.cos(b), s * np.sin(b)], 1)
    db, do = (gcmfgh.DeviceLayer(synth.Layer.from_rings([x])) for x in (P, Q))
    ids = np.zeros(1, np.int32)
    got = []
    try:
        engine.set_precision(True)
        for fused in (1, 0):
            engine.set_tuning(fused_emit=fused)
            engine.clip_batch(db, do, ids, ids)
            got.append(engine.clip_result())
    finally:
        engine.set_precision(False)
        engine.set_tuning(fused_emit=1)
    assert got[0].count1[0] > 100
    for f in ("status", "count1", "comp_size", "xy"):
        assert np.array_equal(getattr(got[0], f), getattr(got[1], f)), f
