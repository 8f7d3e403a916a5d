"""Tiles a little narrower than a power of two, placed so that the octree's root cube
begins inside them: it is rounded to a sixteenth of its side, and the first part
of a metre lies beside it.  Terrain with buildings and trees, one tile with points
beside two faces, one beside one, and the same far from the origin; labels by every
kernel against the oracle, a tile in a batch beside one without such points, and
the queries."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

OFFSETS = {"two_faces": (0.7, 0.7, 0.0), "one_face": (0.7, 0.0, 0.0), "other_face": (0.0, 0.9, 0.0),
           "far": (500000.7, 4500000.7, 0.0)}


def _cloud(offset, sign=(1, 1, 1), seed=94):
    from wolkenbase_gb300 import synth
    c = synth.density_tile(24800, seed)
    xyz = np.ascontiguousarray(c.xyz * np.array(sign, np.int32))
    scale = tuple(s * g for s, g in zip(c.scale, sign))
    return synth.Cloud(xyz, scale, offset, 1.0, tuple(np.array(c.minc) + offset), tuple(np.array(c.maxc) + offset))


@pytest.fixture(scope="module", params=sorted(OFFSETS))
def case(request, oracle_mod):
    cloud = _cloud(OFFSETS[request.param])
    o = oracle_mod.run(cloud, canonical_order=True, threads=8)
    lo = np.array(o["root_center"]) - o["root_side"] / 2
    beside = np.any(cloud.decoded()[:, :2] < lo[:2], axis=1)
    assert 100 < beside.sum() < 2000
    return cloud, o, beside


def _check(classifier, O, cloud, o, got, beside):
    """Every label but those of points that the reference decides with another
    point's list (see wrong); those by pointsIn alone."""
    from test_gpu_outside import _wrong
    bad = _wrong(classifier, O, cloud, got)
    assert bad.size == 0, f"{bad.size} labels differ, {np.sum(beside[bad])} of them of points beside the root cube"


@pytest.mark.parametrize("shape", [0, 1, 2, 3, 4])
def test_labels(classifier, oracle_mod, case, shape):
    import wolkenbase_gb300 as wb
    cloud, o, beside = case
    keep = classifier.tuning()
    classifier.set_tuning(shape=shape)
    try:
        got = classifier.classify_cloud(cloud, wb.Params())
    finally:
        classifier.set_tuning(shape=keep["shape"])
    _check(classifier, oracle_mod, cloud, o, got, beside)
    assert np.array_equal(classifier.tiles()["n_points"], o["tiles"]["n_points"])
    assert np.array_equal(classifier.tiles()["hyperboloid_size"], o["tiles"]["h_final"])


def test_labels_with_margins(classifier, oracle_mod, case):
    import wolkenbase_gb300 as wb
    cloud, o, beside = case
    classifier.build(cloud)
    classifier.scan(wb.Params())
    plain = classifier.classify(wb.Params()).copy()
    got, _ = classifier.classify_margins(wb.Params())
    assert np.array_equal(got, plain)
    _check(classifier, oracle_mod, cloud, o, got, beside)


def test_labels_of_the_exact_pass(classifier, oracle_mod):
    import wolkenbase_gb300 as wb
    cloud = _cloud(OFFSETS["two_faces"], (-1, 1, 1))
    o = oracle_mod.run(cloud, canonical_order=True, threads=8)
    got = classifier.classify_cloud(cloud, wb.Params())
    _check(classifier, oracle_mod, cloud, o, got, np.zeros(cloud.n, bool))


def test_batch_of_both_kinds(classifier, cuda_lib_path):
    import wolkenbase_gb300 as wb
    from wolkenbase_gb300 import _lib, synth
    clouds = [synth.density_tile(9000, 95), _cloud(OFFSETS["two_faces"]), synth.density_tile(3000, 96), _cloud(OFFSETS["far"], seed=97)]
    srv = wb.Server(0, prep_slots=4, flush=_lib.WB_FLUSH_FULL)
    try:
        got = srv.classify_batch(clouds, wb.Params())
    finally:
        srv.close()
    for c, g in zip(clouds, got):
        assert np.array_equal(np.asarray(g), classifier.classify_cloud(c, wb.Params()))


def test_precision_mode(classifier, case):
    """FP32 decisions: at most a few labels other than the exact ones."""
    import wolkenbase_gb300 as wb
    from wolkenbase_gb300 import _lib
    cloud = case[0]
    exact = classifier.classify_cloud(cloud, wb.Params()).copy()
    classifier.set_precision(_lib.WB_PRECISION_FP32)
    try:
        got = classifier.classify_cloud(cloud, wb.Params())
    finally:
        classifier.set_precision(_lib.WB_PRECISION_EXACT)
    assert np.sum(got != exact) <= 3


def test_queries(classifier, oracle_mod, case):
    cloud, _, beside = case
    d = cloud.decoded()
    classifier.build(cloud)
    oracle_mod.run(cloud, canonical_order=True, phases=1, keep=True)
    try:
        r = np.random.default_rng(98)
        pick = np.concatenate([r.choice(np.nonzero(beside)[0], 12), r.integers(0, cloud.n, 12)])
        for j in pick:
            for kind, v, rad in ((1, tuple(d[j, :2]), 0.8), (1, tuple(d[j, :2]), 4.0), (2, tuple(d[j] + [0, 0, 1.5]), 0.2)):
                assert np.array_equal(classifier.find_blocks(kind, v, rad, 1.0), oracle_mod.find_blocks(kind, v, rad, 1.0))
                for srt in (False, True):
                    assert np.array_equal(classifier.points_in(kind, v, rad, 1.0, sorted=srt),
                                          oracle_mod.points_in(kind, v, rad, 1.0, sorted=srt))
    finally:
        oracle_mod.reset()
