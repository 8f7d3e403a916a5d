"""The octree build's sort and scans at the sizes where they can go wrong, against
the oracle: leaf cubes, the point -> leaf map and the store order equal.  Clouds
around the sizes of the sort's and the scans' tiles, stacks and lines of points
too long for a thread or a block to order, points all on cell boundaries,
many duplicates, and columns of any size (an outlier that puts all others in
one)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _cloud(xyz, scale=(0.001, 0.001, 0.001)):
    from wolkenbase_gb300 import synth
    c = synth.Cloud(np.ascontiguousarray(xyz, np.int32), scale, (0.0, 0.0, 0.0), 1.0, (0, 0, 0), (0, 0, 0))
    d = c.decoded()
    c.minc, c.maxc = tuple(map(float, d.min(axis=0))), tuple(map(float, d.max(axis=0)))
    return c


def _random(n, seed, side=20000, height=2000):
    r = np.random.default_rng(seed)
    return np.stack([r.integers(0, side, n), r.integers(0, side, n), r.integers(0, height, n)], 1)


def _stack(n, seed):
    # n points within a few millimetres: the sorted bits cannot tell them apart
    r = np.random.default_rng(seed)
    a = np.stack([r.integers(5000, 5004, n), r.integers(5000, 5004, n), r.integers(100, 100 + max(2, n // 4), n)], 1)
    a = np.concatenate([a, _random(3000, seed + 1)])
    return a[r.permutation(len(a))]


def _dups(n, seed):
    a = _random(n, seed)
    r = np.random.default_rng(seed)
    return a[r.integers(0, n // 20, n)]


def _outlier(n, seed):
    a = _random(n, seed, side=3000, height=800)
    a[n // 2] = (300_000, 300_000, 400)
    return a


CASES = {f"n{n}": _random(n, n) for n in (1, 2, 537, 538, 539, 1023, 1025, 4095, 4096, 4097, 8193, 40000)}
CASES.update({"stack30": _stack(30, 1), "stack400": _stack(400, 2), "stack2000": _stack(2000, 3),
              "stack9000": _stack(9000, 4), "boundaries": _random(6000, 5, side=160, height=16) * 125,
              "dups": _dups(9000, 6), "outlier600": _outlier(600, 7), "outlier5000": _outlier(5000, 8)})


@pytest.mark.parametrize("name", sorted(CASES))
def test_octree_and_labels_match_oracle(classifier, oracle_mod, name):
    import wolkenbase_gb300 as wb
    cloud = _cloud(CASES[name])
    if name == "n1":
        cloud.minc, cloud.maxc = tuple(v - 1.0 for v in cloud.minc), tuple(v + 1.0 for v in cloud.maxc)
    o = oracle_mod.run(cloud, canonical_order=True, threads=8)
    classifier.build(cloud)
    cs, first, count = classifier.leaves()
    stored = o["leaf"] >= 0
    assert classifier.info()["n_leaves"] == o["n_leaves"]
    assert np.array_equal(cs, o["leaves"]) and np.array_equal(count.astype(np.int64), o["leaf_count"])
    assert np.array_equal(classifier.point_leaf()[stored].astype(np.int64), o["leaf"][stored])
    order = classifier.store_order()
    assert np.array_equal(np.sort(order), np.nonzero(stored)[0])
    for f, k in zip(first, count):
        assert np.all(np.diff(order[f:f + k].astype(np.int64)) > 0)
    classifier.scan(wb.Params())
    got = classifier.classify(wb.Params())
    assert np.array_equal(got[stored], o["cls"][stored])
