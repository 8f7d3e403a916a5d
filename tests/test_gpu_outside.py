"""Clouds whose header box is smaller than their points, against the oracle: the
tiles' counts and every label, whichever kernel decides them.  Clumps of points
lie beside, above and below the octree's root cube; the reference takes such a
point with its block, whose cube lies at the root cube's face, so a neighbour
counts that the query's shape itself does not hold."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _points(seed, kinds):
    r = np.random.default_rng(seed)
    side = [7.8, 3.9, 15.5][seed % 3]   # the root cube is a little larger
    u = lambda n, lo, hi: r.uniform(lo, hi, n)
    ground = np.stack([u(1500, 0, side), u(1500, 0, side), 0.1 * side + u(1500, -0.05, 0.05)], 1)
    high = np.stack([u(400, 0, side), u(400, 0, side), u(400, 0.2, 1.0) * side], 1)
    edge = np.stack([side - u(150, 0, 0.1) * side, u(150, 0, side), u(150, 0.3, 1.0) * side], 1)
    parts = [ground, high, edge, edge[:, [1, 0, 2]]]
    for k in kinds:
        m = int(r.integers(600, 2500))
        a, b = u(1, 0, 0.8)[0] * side, u(1, 0, 0.5)[0] * side
        # lower case: from the root cube's face on, upper case: farther than any query's reach
        far = side * (1 + 10.0 ** (u(m, -2, 0.7) if k.islower() else u(m, 1.0, 1.5)))
        p, q = a + u(m, 0, 0.2) * side, b + u(m, 0, 0.2) * side
        parts.append({"x": np.stack([far, p, q], 1), "y": np.stack([p, far, q], 1), "w": np.stack([side - far, p, q], 1),
                      "c": np.stack([far, far[::-1], q], 1), "a": np.stack([p, a + (q - b), far], 1),
                      "b": np.stack([p, q, -far], 1)}[k.lower()])
    d = np.concatenate(parts)
    return d[r.permutation(len(d))], side


def _cloud(seed, kinds, sign=(1, 1, 1), head=1.0):
    """head: the part of the points' box that the header gives."""
    from wolkenbase_gb300 import synth
    d, side = _points(seed, kinds)
    scale = tuple(0.001 * s for s in sign)
    xyz = np.rint(d / np.array(scale)).astype(np.int32)
    return synth.Cloud(np.ascontiguousarray(xyz), scale, (0.0, 0.0, 0.0), 1.0, (0.0,) * 3, (head * side,) * 3)


CLOUDS = {f"{kinds or 'none'}_{seed}_{head}": (seed, kinds, head)
          for kinds, seeds, head in (("x", (0, 1), 1.0), ("y", (2,), 1.0), ("w", (3,), 1.0), ("c", (4,), 1.0), ("a", (5, 6), 1.0),
                                     ("b", (7,), 1.0), ("xywcab", (8, 9, 10), 1.0), ("", (0, 1, 2), 0.6), ("xa", (3, 4), 0.6),
                                     ("X", (0, 1, 2, 3), 1.0), ("W", (4,), 1.0), ("XYW", (5, 6, 7), 1.0), ("A", (8,), 1.0), ("XA", (9, 10), 0.6))
          for seed in seeds}


def _wrong(classifier, O, cloud, got):
    """Stored points with another label than the reference's.  The reference tries
    the list of the point before first, so beside the root cube a label can depend
    on which point that was; where labels differ, the points that pointsIn alone
    returns decide (their integer directions' largest gap against 144 degrees)."""
    o = O.run(cloud, canonical_order=True, threads=8, keep=True)
    try:
        stored = np.zeros(cloud.n, bool)
        stored[classifier.store_order()] = True
        differ = np.nonzero((got != o["cls"]) & stored)[0]
        if not differ.size:
            return differ
        assert set(got[differ].tolist()) <= {1, 2} and set(o["cls"][differ].tolist()) <= {1, 2}
        t, d = o["tiles"], cloud.decoded()
        owner = np.full(cloud.n, -1)
        for k in np.nonzero(t["n_points"])[0]:
            cx = o["snake_center"][0] + (t["ex"][k] - t["ey"][k] / 2) * o["spacing"]
            cy = o["snake_center"][1] + t["ey"][k] * 0.86602540378443864676372317 * o["spacing"]
            owner[O.points_in(1, (cx, cy), o["spacing"] * 41 / 71)] = k
        wrong = []
        for j in differ:
            q = O.points_in(2, tuple(d[j]), t["h_final"][owner[j]])
            v = d[q] - d[j]
            v = v[(v[:, 0] != 0) | (v[:, 1] != 0)]
            u = np.unique(O.atan2i(v[:, 1], v[:, 0]).astype(np.int64) & 0x7fffffff)
            gap = np.max((np.roll(u, -1) - u) & 0x7fffffff) if u.size > 1 else 1 << 31
            if got[j] != (1 if gap < 0x33333333 else 2):
                wrong.append(j)
        return np.array(wrong, int)
    finally:
        O.reset()


@pytest.mark.parametrize("name", sorted(CLOUDS))
def test_tiles(classifier, oracle_mod, name):
    import wolkenbase_gb300 as wb
    seed, kinds, head = CLOUDS[name]
    cloud = _cloud(seed, kinds, head=head)
    o = oracle_mod.run(cloud, canonical_order=True, threads=8, phases=2)
    classifier.build(cloud)
    classifier.scan(wb.Params())
    t = classifier.tiles()
    assert np.array_equal(t["n_points"], o["tiles"]["n_points"])
    assert np.array_equal(t["hyperboloid_size"], o["tiles"]["h_final"])


@pytest.mark.parametrize("shape", [0, 1, 2, 4])
@pytest.mark.parametrize("name", sorted(CLOUDS))
def test_labels(classifier, oracle_mod, name, shape):
    """Point groups (0-2) and the one-point kernel (4)."""
    import wolkenbase_gb300 as wb
    seed, kinds, head = CLOUDS[name]
    cloud = _cloud(seed, kinds, head=head)
    keep = classifier.tuning()
    classifier.set_tuning(shape=shape)
    try:
        got = classifier.classify_cloud(cloud, wb.Params())
    finally:
        classifier.set_tuning(shape=keep["shape"])
    bad = _wrong(classifier, oracle_mod, cloud, got)
    assert bad.size == 0, f"{bad.size} of {cloud.n} labels differ, e.g. {bad[:8].tolist()}"


@pytest.mark.parametrize("name", sorted(CLOUDS))
def test_labels_with_margins(classifier, oracle_mod, name):
    """The column groups and bins."""
    import wolkenbase_gb300 as wb
    seed, kinds, head = CLOUDS[name]
    cloud = _cloud(seed, kinds, head=head)
    classifier.build(cloud)
    classifier.scan(wb.Params())
    got, _ = classifier.classify_margins(wb.Params())
    bad = _wrong(classifier, oracle_mod, cloud, got)
    assert bad.size == 0, f"{bad.size} of {cloud.n} labels differ, e.g. {bad[:8].tolist()}"


@pytest.mark.parametrize("sign", [(-1, 1, 1), (1, 1, -1)])
@pytest.mark.parametrize("name", sorted(CLOUDS))
def test_labels_of_the_exact_pass(classifier, oracle_mod, name, sign):
    """A scale below zero: the exact pass decides every point."""
    import wolkenbase_gb300 as wb
    seed, kinds, head = CLOUDS[name]
    cloud = _cloud(seed, kinds, sign, head)
    got = classifier.classify_cloud(cloud, wb.Params())
    bad = _wrong(classifier, oracle_mod, cloud, got)
    assert bad.size == 0, f"{bad.size} of {cloud.n} labels differ, e.g. {bad[:8].tolist()}"


def _rough(seed, sign, head, n, side):
    from wolkenbase_gb300 import synth
    r = np.random.default_rng(seed)
    d = np.stack([r.uniform(0, side, n), r.uniform(0, side, n), r.uniform(0, 0.1 * side, n)], 1)
    scale = tuple(0.001 * s for s in sign)
    lo = 0.5 * (side - head)
    return synth.Cloud(np.rint(d / np.array(scale)).astype(np.int32), scale, (0.0, 0.0, 0.0), 1.0, (lo, lo, 0.0),
                       (side - lo, side - lo, 0.1 * side))


@pytest.mark.parametrize("sign", [(-1, 1, 1), (1, 1, -1)])
@pytest.mark.parametrize("n", [2000, 60000])
def test_exact_pass_beside_the_grid(classifier, oracle_mod, n, sign):
    """Points up to fourteen columns beside the header's box and inside the root
    cube; their nearest neighbours are in the grid's edge columns."""
    import wolkenbase_gb300 as wb
    cloud = _rough(3, sign, 2.05, n, 4.0)
    got = classifier.classify_cloud(cloud, wb.Params())
    bad = _wrong(classifier, oracle_mod, cloud, got)
    assert bad.size == 0, f"{bad.size} of {cloud.n} labels differ, e.g. {bad[:8].tolist()}"


@pytest.mark.parametrize("kernel", ["groups", "points", "bins", "exact"])
def test_reach_of_many_grid_widths(classifier, oracle_mod, kernel):
    """A slope of 1e-4: half a metre of height reaches six kilometres, the grid six metres."""
    import wolkenbase_gb300 as wb
    cloud = _rough(4, (-1, 1, 1) if kernel == "exact" else (1, 1, 1), 6.0, 1500, 6.0)
    p = dict(max_slope=1e-4)
    o = oracle_mod.run(cloud, canonical_order=True, threads=8, **p)
    keep = classifier.tuning()
    classifier.set_tuning(shape=4 if kernel == "points" else 0)
    try:
        classifier.build(cloud)
        classifier.scan(wb.Params(**p))
        got = classifier.classify_margins(wb.Params(**p))[0] if kernel == "bins" else classifier.classify(wb.Params(**p))
    finally:
        classifier.set_tuning(shape=keep["shape"])
    assert np.array_equal(got, o["cls"])
