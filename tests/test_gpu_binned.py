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
