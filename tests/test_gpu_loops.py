"""Tracing by loops (warp and block labelling): degenerate pairs, whose flags, chains, split
vertices and non-closing walks take every branch of it, against the oracle."""
import numpy as np
import pytest

import pyoracle
from gcmfgh import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("union", [False, True])
@pytest.mark.parametrize("exact", [False, True])
@pytest.mark.parametrize("mid_label", [0, 1 << 20])
def test_degenerate_pairs(engine, union, exact, mid_label):
    import gcmfgh
    # lattice stars with few distinct coordinates: shared vertices, collinear overlaps,
    # bouncing and crossing chains; and the workload's own classes
    rng = np.random.default_rng(31)
    pairs = synth.degeneracy_pairs(31, 300, 4, 400)[1]
    for k in range(500):
        q = 0.5 ** rng.integers(0, 3)
        P, Q = (np.round(synth._star(rng, int(rng.integers(4, 60)), 0.0, 0.0, 6.0, 0.3, 1.0) / q) * q for _ in range(2))
        pairs.append((P, Q if k % 5 else np.roll(P, int(rng.integers(len(P))), 0)))
    base, ovl = (synth.Layer.from_rings([p[i] for p in pairs]) for i in (0, 1))
    ids = np.arange(len(pairs), dtype=np.int32)
    db, do = gcmfgh.DeviceLayer(base), gcmfgh.DeviceLayer(ovl)
    try:
        engine.set_tuning(tile_label=0, mid_label=mid_label, big_label=1 << 24)
        engine.set_params(1e-7, 1e-7, union)
        engine.set_precision(exact)
        engine.clip_batch(db, do, ids, ids)
        r = engine.clip_result()
    finally:
        engine.set_tuning(tile_label=96, mid_label=1 << 10, big_label=1 << 18)
        engine.set_params(1e-7, 1e-7, False)
        engine.set_precision(False)
    o = pyoracle.clip_batch(base, ovl, ids, ids, union=union, exact=exact)
    assert np.array_equal(r.status, o.status)
    assert np.array_equal(r.ncomp, o.ncomp)
    assert np.array_equal(r.comp_size, o.comp_size)
    assert np.array_equal(r.xy, o.xy)
