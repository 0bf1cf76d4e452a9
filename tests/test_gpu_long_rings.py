"""Block-per-pair stages, edge insertion classes, sort and scan forms and pairs per warp, at
the sizes where one form hands over to the next, against the oracle (bit for bit)."""
import numpy as np
import pytest

import pyoracle
from gcmfgh import synth

pytestmark = pytest.mark.gpu


def _clip_equal(r, o):
    assert np.array_equal(r.status, o.status)
    assert np.array_equal(r.count1[r.status != 2], o.count1[o.status != 2])
    assert np.array_equal(r.ncomp, o.ncomp)
    assert np.array_equal(r.comp_size, o.comp_size)
    assert np.array_equal(r.xy, o.xy)


def _layers(sizes_b, sizes_o, seed):
    rng = np.random.default_rng(seed)
    out = []
    for sizes in (sizes_b, sizes_o):
        counts = np.array(sizes)
        centres = rng.uniform(0.0, 30.0, size=(len(counts), 2))
        out.append(synth.star_layer(rng, counts, centres, rng.uniform(4.0, 14.0, size=len(counts))))
    return out


# around 1,024 (an MBR's block), 2,048 (a pair's block), 4,096 (a copied piece), with small ones between
SIZES = [4, 1023, 1024, 1025, 7, 64, 65, 2044, 2047, 2048, 2049, 12, 4095, 4097, 128, 129, 9001]


@pytest.mark.parametrize("union", [False, True])
@pytest.mark.parametrize("two_pass,f32", [(False, 1), (True, 1), (False, 3)])
def test_join_and_clip_of_long_rings(engine, union, two_pass, f32):
    import gcmfgh
    # enough pairs for the listed form of the clip's edge filter (more than 296 of them)
    base, ovl = _layers(SIZES + [20] * 30, SIZES[::-1] + [9] * 30, 5)
    oj = pyoracle.join(base, ovl)
    assert int(oj.clip.sum()) > 296
    db, do = gcmfgh.DeviceLayer(base), gcmfgh.DeviceLayer(ovl)
    engine.set_tuning(sweep_two_pass=two_pass, f32_filter=f32)
    engine.set_params(1e-7, 1e-7, union)
    try:
        engine.join(db, do)
        for name, want in (("b", oj.b), ("o", oj.o), ("pip_flag", oj.pip_flag), ("join_flag", oj.join_flag),
                           ("bE", oj.bE), ("oE", oj.oE), ("seg_flag", oj.seg_flag), ("clip", oj.clip)):
            assert np.array_equal(engine.join_field(name), want), name
        engine.clip_joined(db, do)
        r = engine.clip_result()
        cb, co = engine.join_field("clip_b"), engine.join_field("clip_o")
        _clip_equal(r, pyoracle.clip_batch(base, ovl, cb, co, union=union))
        engine.clip_batch(db, do, cb, co)                     # the filter's own edge lists
        _clip_equal(engine.clip_result(), r)
        engine.clip_batch(db, do, cb[:290], co[:290])         # a block per pair
        _clip_equal(engine.clip_result(), pyoracle.clip_batch(base, ovl, cb[:290], co[:290], union=union))
    finally:
        engine.set_tuning(sweep_two_pass=False, f32_filter=1)
        engine.set_params(1e-7, 1e-7, False)


@pytest.mark.parametrize("crossings", [7, 8, 9, 31, 32, 33, 64, 65, 511, 512, 513, 1100])
def test_insertions_per_edge(engine, crossings):
    """A strip crossed by a comb: about `crossings` insertions on each long edge."""
    import gcmfgh
    n = (crossings + 1) // 2
    top = [(2.0 * i + d, y) for i in range(n) for d, y in ((0.0, -1.0), (0.5, 2.0), (1.0, -1.0))]
    comb = np.array(top + [(2.0 * n + 1.0, -3.0), (-1.0, -3.0)])[::-1]
    strip = np.array([(-5.0, 0.0), (2.0 * n + 5.0, 0.1), (2.0 * n + 5.0, 1.0), (-5.0, 0.9)])
    base, ovl = synth.Layer.from_rings([comb, strip]), synth.Layer.from_rings([strip, comb])
    ids = np.array([0, 1], np.int32)
    engine.clip_batch(gcmfgh.DeviceLayer(base), gcmfgh.DeviceLayer(ovl), ids, ids)
    _clip_equal(engine.clip_result(), pyoracle.clip_batch(base, ovl, ids, ids))


@pytest.mark.parametrize("exact", [False, True])
def test_long_loop_by_the_grid(engine, exact):
    """One loop of several thousand segments (decided over nodes) among short ones."""
    import gcmfgh
    rng = np.random.default_rng(11)
    rings = []
    for n, k in ((3600, 900), (2800, 700)):
        a = np.sort(rng.uniform(0.0, 2.0 * np.pi, n))
        r = 10.0 + np.sin(k * a) + rng.uniform(-0.2, 0.2, n)
        rings.append(np.stack([r * np.cos(a), r * np.sin(a)], 1))
    base, ovl = synth.Layer.from_rings(rings[:1]), synth.Layer.from_rings(rings[1:])
    ids = np.zeros(1, np.int32)
    try:
        engine.set_tuning(big_label=0)
        engine.set_precision(exact)
        for union in (False, True):
            engine.set_params(1e-7, 1e-7, union)
            engine.clip_batch(gcmfgh.DeviceLayer(base), gcmfgh.DeviceLayer(ovl), ids, ids)
            _clip_equal(engine.clip_result(), pyoracle.clip_batch(base, ovl, ids, ids, union=union, exact=exact))
    finally:
        engine.set_tuning(big_label=1 << 18)
        engine.set_precision(False)
        engine.set_params(1e-7, 1e-7, False)


# one block, one kernel per pass (to 512 tiles of 2,048), three kernels per pass
@pytest.mark.parametrize("n", [3, 4095, 4096, 4097, 512 * 2048, 512 * 2048 + 1])
@pytest.mark.parametrize("bits", [8, 33, 64])
def test_sort_forms(engine, n, bits):
    import torch
    rng = np.random.default_rng(n + bits)
    keys = rng.integers(0, 1 << 63, size=n, dtype=np.int64).view(np.uint64) * np.uint64(2) + np.uint64(1)
    keys[rng.integers(0, n, size=n // 3)] = keys[0]           # equal keys: stable in the values
    dk = torch.from_numpy(keys.view(np.int64).copy()).cuda()
    dv = torch.from_numpy(np.arange(n, dtype=np.int32)).cuda()
    engine.radix_sort_u64(dk, dv, bits)
    low = ((bits + 7) // 8) * 8
    order = np.argsort(keys & np.uint64((1 << low) - 1), kind="stable")
    assert np.array_equal(dk.cpu().numpy().view(np.uint64), keys[order])
    assert np.array_equal(dv.cpu().numpy(), order.astype(np.int32))


def test_multi_pairs_sharing_a_warp(engine):
    """More pairs than warps to spare: several pairs of rings with holes per warp."""
    import gcmfgh
    few = synth.holed_pairs(3, 40, 3, 8)
    few += [([np.array([[0.0, 0.0], [1.0, 0.0], [0.0, 1.0]])], [np.array([[0.5, 0.1], [2.0, 0.1], [0.5, 2.0]])])] * 20
    pairs = few * 170                                         # 10,200 pairs: two per warp
    engine.clip_multi_batch(pairs)
    many = engine.clip_result()
    engine.clip_multi_batch(few)                              # one per warp
    one = engine.clip_result()
    assert np.array_equal(many.status, np.tile(one.status, 170))
    assert np.array_equal(many.ncomp, np.tile(one.ncomp, 170))
    assert np.array_equal(many.comp_size, np.tile(one.comp_size, 170))
    assert np.array_equal(many.xy, np.tile(one.xy, 170))
