"""The octree of clouds of a few centimetres far from the origin, where a
coordinate's rounding is as wide as a level-21 cell or wider, against the oracle:
leaf cubes, the point -> leaf map, the survivors and their order equal.  Points
crowd around the root cube's centre planes and decode to the same doubles in
runs, so a cell that is one off changes the leaves or keeps a duplicate."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# offset, scale, unit, half the extent in record units, half the crowd's
CASES = {
    "side_8_at_4.5e6": (4.5e6, 1e-3, 1.0, 3900, 900),
    "quarter_at_1e9": (1e9, 1e-7, 0.3048, 2_000_000, 40),
    "eighth_at_6.5e9": (6.5e9, 1e-6, 1.0, 60_000, 40),
    "dups_at_6.5e9": (6.5e9, 1e-8, 1.0, 6_000_000, 400),
    "two_at_1.7e7": (1.848785e7, 1.7e-6, 0.906, 500_000, 40),
    "half_at_4e8": (4e8, 1e-6, 0.9, 250_000, 40),
}


@pytest.mark.parametrize("name", sorted(CASES))
def test_octree_far_from_the_origin(classifier, oracle_mod, name):
    from wolkenbase_gb300 import synth
    offset, scale, unit, half, crowd = CASES[name]
    r = np.random.default_rng(11)
    wide = r.integers(-half, half + 1, (3000, 3))
    near = r.integers(-crowd, crowd + 1, (6000, 3))
    lines = r.integers(-half, half + 1, (3000, 3))
    lines[:, 1:] = r.integers(-crowd, crowd + 1, (3000, 2))
    xyz = np.concatenate([wide, near, lines])
    xyz = xyz[r.permutation(len(xyz))].astype(np.int32)
    lo, hi = (offset + scale * float(v) for v in (-half, half))
    cloud = synth.Cloud(np.ascontiguousarray(xyz), (scale,) * 3, (offset,) * 3, unit, (lo,) * 3, (hi,) * 3)
    o = oracle_mod.run(cloud, canonical_order=True, phases=1)
    classifier.build(cloud)
    cs, first, count = classifier.leaves()
    stored = o["leaf"] >= 0
    assert classifier.info()["n_leaves"] == o["n_leaves"]
    assert np.array_equal(cs, o["leaves"]) and np.array_equal(count.astype(np.int64), o["leaf_count"])
    assert np.array_equal(classifier.point_leaf()[stored].astype(np.int64), o["leaf"][stored])
    assert np.array_equal(np.sort(classifier.store_order()), np.nonzero(stored)[0])
