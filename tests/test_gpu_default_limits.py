"""The one-thread labelling's limit that an engine chooses by the batch: kept when another
threshold is set, and the same results on both sides of its two borders."""
import numpy as np
import pytest

import pyoracle
from gcmfgh import synth

pytestmark = pytest.mark.gpu

CHOSEN = {1: 0, (1 << 15) - 1: 0, 1 << 15: 32, (1 << 16) - 1: 32, 1 << 16: 96, 1 << 20: 96}


def test_one_threshold_leaves_the_others():
    import gcmfgh
    base, ovl = synth.small_join(seed=0, n=20)
    eng = gcmfgh.Engine(0)
    try:
        db, do = gcmfgh.DeviceLayer(base), gcmfgh.DeviceLayer(ovl)

        def limits():
            return {n: eng.tuning_for(db, do, n)["tile_label"] for n in CHOSEN}

        assert limits() == CHOSEN
        for other in ("bin_grid", "big_label", "mid_label", "wide_label"):
            eng.set_tuning(**{other: 1 << 12})
            assert limits() == CHOSEN
            assert eng.tuning_for(db, do, 1)[other] == 1 << 12
        eng.set_tuning(tile_label=64)
        assert set(limits().values()) == {64}
        eng.set_tuning(defaults=True)
        assert limits() == CHOSEN
        assert eng.tuning_for(db, do, 1)["bin_grid"] == 1 << 16
    finally:
        eng.close()


@pytest.mark.parametrize("n", [(1 << 15) - 1, 1 << 15, (1 << 16) - 1, 1 << 16])
@pytest.mark.parametrize("union,exact", [(False, False), (True, True)])
def test_batches_at_the_borders(n, union, exact):
    import gcmfgh
    few = synth.random_star_pairs(9, 600, 3, 40) + synth.degeneracy_pairs(9, 400, 4, 60)[1]
    base, ovl = (synth.Layer.from_rings([p[i] for p in few]) for i in (0, 1))
    ids = (np.arange(n) % len(few)).astype(np.int32)
    eng = gcmfgh.Engine(0, union=union)
    try:
        eng.set_precision(exact)
        eng.clip_batch(gcmfgh.DeviceLayer(base), gcmfgh.DeviceLayer(ovl), ids, ids)
        r = eng.clip_result()
    finally:
        eng.close()
    o = pyoracle.clip_batch(base, ovl, ids, ids, union=union, exact=exact)
    assert np.array_equal(r.status, o.status)
    assert np.array_equal(r.comp_size, o.comp_size)
    assert np.array_equal(r.xy, o.xy)
