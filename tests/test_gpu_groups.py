"""The classify's point groups (runs of 32 points, octets, super-cells) and
their open arcs at the sizes and shapes where they can go wrong, against the
oracle: every label equal.  Clouds with a handful of points, one more and one
fewer than a group, several groups per super-cell, columns of very many points,
different scales per axis, a thickness, slopes other than one, directions that
coincide (points on a lattice and on lines), and the one-point kernel on the
same clouds."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _cloud(xyz, scale=(0.001, 0.001, 0.001), offset=(0.0, 0.0, 0.0)):
    from wolkenbase_gb300 import synth
    c = synth.Cloud(np.ascontiguousarray(xyz, np.int32), scale, offset, 1.0, (0, 0, 0), (0, 0, 0))
    d = c.decoded()
    c.minc, c.maxc = tuple(map(float, d.min(axis=0))), tuple(map(float, d.max(axis=0)))
    return c


def _random(n, seed, side=3000, height=400):
    r = np.random.default_rng(seed)
    return np.stack([r.integers(0, side, n), r.integers(0, side, n), r.integers(0, height, n)], 1)


def _lattice(seed):
    # directions and heights that repeat exactly, with a few raised points
    x, y = np.meshgrid(np.arange(0, 3000, 100), np.arange(0, 3000, 100))
    z = (x // 7 + (x * y) % 3 * 20).astype(np.int64)
    p = np.stack([x.ravel(), y.ravel(), z.ravel()], 1)
    p[:: 17, 2] += 900 + seed
    return p


def _pillar(seed):
    # thousands of points above each other, and the ground around them
    r = np.random.default_rng(seed)
    a = np.stack([r.integers(1480, 1520, 4000), r.integers(1480, 1520, 4000), r.integers(0, 8000, 4000)], 1)
    return np.concatenate([a, _random(1500, seed + 1, height=60)])


CASES = {
    "one": (np.array([[5, 7, 9], [6, 7, 30]]), {}, {}),
    "n31": (_random(31, 1), {}, {}),
    "n32": (_random(32, 2), {}, {}),
    "n33": (_random(33, 3), {}, {}),
    "n577": (_random(577, 4), {}, {}),
    "sparse": (_random(900, 5, side=90000, height=3000), {}, {}),
    "flat": (_random(3000, 6, height=3), {}, {}),
    "rough": (_random(3000, 7, height=4000), {}, {}),
    "lattice": (_lattice(1), {}, {}),
    "pillar": (_pillar(8), {}, {}),
    "thick": (_random(2000, 9, height=900), {}, dict(thickness=0.35)),
    "thin": (_random(2000, 10, height=900), {}, dict(thickness=-0.2)),
    "slope": (_random(2000, 11, height=900), {}, dict(max_slope=0.4)),
    "steep": (_random(2000, 12, height=2500), {}, dict(max_slope=2.5, tile_size=0.6)),
    "axes": (_random(2000, 13) * [1, 4, 10], dict(scale=(0.001, 0.00025, 0.0001)), {}),
    "far": (_random(2000, 14), dict(offset=(500000.0, 4500000.0, 1500.0)), dict(min_hyp_size=0.5)),
}


@pytest.mark.parametrize("shape", [0, 1, 2, 4])
@pytest.mark.parametrize("name", sorted(CASES))
def test_labels_match_oracle(classifier, oracle_mod, name, shape):
    import wolkenbase_gb300 as wb
    xyz, ckw, pkw = CASES[name]
    cloud = _cloud(xyz, **ckw)
    o = oracle_mod.run(cloud, canonical_order=True, threads=8, **pkw)
    keep = classifier.tuning()
    classifier.set_tuning(shape=shape)
    try:
        got = classifier.classify_cloud(cloud, wb.Params(**pkw))
    finally:
        classifier.set_tuning(shape=keep["shape"])
    stored = np.zeros(cloud.n, bool)
    stored[classifier.store_order()] = True
    bad = np.nonzero((got != o["cls"]) & stored)[0]
    assert bad.size == 0, f"{bad.size} of {cloud.n} labels differ, e.g. {bad[:8].tolist()}"


def test_empty_cloud_after_another(classifier):
    """A cloud without records leaves no group of the one before."""
    import wolkenbase_gb300 as wb
    cloud = _cloud(_random(3000, 15))
    classifier.classify_cloud(cloud)
    from wolkenbase_gb300 import synth
    empty = synth.Cloud(np.zeros((0, 3), np.int32), cloud.scale, cloud.offset, 1.0, cloud.minc, cloud.maxc)
    assert classifier.classify_cloud(empty, wb.Params()).size == 0
    again = classifier.classify_cloud(cloud)
    assert np.array_equal(again, classifier.classify_cloud(cloud))
