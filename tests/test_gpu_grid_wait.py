"""The grid-wide labelling's barrier: a wait without progress ends the call with an error and
leaves the engine usable; a member that works alone for longer than the wait does not."""
import numpy as np
import pytest

import pyoracle
from gcmfgh import synth

pytestmark = pytest.mark.gpu

DEV_TIMEOUT = 4
WAIT = 1 << 26


def _equal(a, b):
    return (np.array_equal(a.status, b.status) and np.array_equal(a.comp_size, b.comp_size)
            and np.array_equal(a.xy, b.xy))


def _layers(rings_p, rings_q):
    import gcmfgh
    base, ovl = synth.Layer.from_rings(rings_p), synth.Layer.from_rings(rings_q)
    return base, ovl, gcmfgh.DeviceLayer(base), gcmfgh.DeviceLayer(ovl), np.arange(len(rings_p), dtype=np.int32)


@pytest.mark.parametrize("exact", [False, True])
def test_wait_that_runs_out(exact):
    """No polls at all: some block gives up at some barrier of the first pairs."""
    import gcmfgh
    rng = np.random.default_rng(4)
    pairs = synth.degeneracy_pairs(5, 40, 4, 300)[1]
    pairs += [tuple(synth._star(rng, n, 0.0, 0.0, 9.0, 0.3, 1.0) for n in (3000, 2500)) for _ in range(3)]
    base, ovl, db, do, ids = _layers([p for p, _ in pairs], [q for _, q in pairs])
    want = pyoracle.clip_batch(base, ovl, ids, ids, exact=exact)
    eng = gcmfgh.Engine(0)
    try:
        eng.set_precision(exact)
        for _ in range(3):
            eng.set_tuning(big_label=0, grid_wait=0)
            with pytest.raises(gcmfgh.GcmfghError):
                eng.clip_batch(db, do, ids, ids)
            assert eng.last_device_error() == DEV_TIMEOUT
            eng.set_tuning(grid_wait=WAIT)
            eng.clip_batch(db, do, ids, ids)
            assert _equal(eng.clip_result(), want)
    finally:
        eng.close()


def _chains(n):
    """Two strips that share every other piece of their lower side (a chain each); one touches a
    vertex of the other twice, so that the chains are resolved by one member."""
    x = np.arange(n + 1, dtype=np.float64)
    P = np.concatenate([np.stack([x, np.zeros(n + 1)], 1), [[n, 5.0], [n / 2, 5.0], [0.0, 5.0]]])
    low = []
    for i in range(0, n, 4):
        low += [(i, 0.0), (i + 1.0, 0.0), (i + 2.0, 0.0), (i + 2.5, -1.0), (i + 3.5, -1.0)]
    top = [(n / 2 + 4.0, 4.0), (n / 2, 5.0), (n / 2 + 2.0, 4.0), (n / 2 - 2.0, 4.0), (n / 2, 5.0), (n / 2 - 4.0, 4.0)]
    Q = np.array([(-1.0, 0.0)] + low + [(n + 1.0, 0.0), (n + 1.0, 4.0)] + top + [(-1.0, 4.0)])
    return P, Q


@pytest.mark.parametrize("union", [False, True])
def test_long_work_of_one_member(union):
    import gcmfgh
    P, Q = _chains(400)
    base, ovl, db, do, ids = _layers([P], [Q])
    eng = gcmfgh.Engine(0, union=union)
    try:
        eng.set_tuning(big_label=0)
        eng.clip_batch(db, do, ids, ids)
        assert _equal(eng.clip_result(), pyoracle.clip_batch(base, ovl, ids, ids, union=union))
        P, Q = _chains(400_000)
        base, ovl, db, do, ids = _layers([P], [Q])
        eng.set_tuning(big_label=1 << 40)                        # a block: no such wait
        eng.clip_batch(db, do, ids, ids)
        want = eng.clip_result()
        assert want.status[0] == 0
        eng.set_tuning(big_label=0, grid_wait=1 << 14)
        eng.clip_batch(db, do, ids, ids)
        assert _equal(eng.clip_result(), want)
    finally:
        eng.close()
