"""Shape queries around the sizes at which their path changes (one block for few
leaves and points, counts and a radix sort beyond), against the oracle: the same
records in the same order, and the count when the caller's buffer is too small."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def built(cuda_lib_path, oracle_mod):
    import wolkenbase_gb300 as wb
    from wolkenbase_gb300 import synth
    cloud = synth.density_tile(120_000, 41, density=900.0)
    clf = wb.Classifier(0)
    clf.build(cloud)
    oracle_mod.run(cloud, canonical_order=True, phases=1, keep=True)
    yield clf, cloud
    oracle_mod.reset()
    clf.close()


@pytest.mark.parametrize("sort", [False, True])
@pytest.mark.parametrize("r", [0.0, 0.02, 0.3, 0.8, 0.9, 1.6, 1.75, 2.6, 5.0, 40.0])
def test_cylinder_of_any_size(built, oracle_mod, r, sort):
    clf, cloud = built
    c = cloud.decoded()[cloud.n // 3]
    got = clf.points_in(1, (c[0], c[1]), r, sorted=sort)
    assert np.array_equal(got, oracle_mod.points_in(1, (c[0], c[1]), r, 1.0, sorted=sort))
    assert np.array_equal(clf.find_blocks(1, (c[0], c[1]), r), oracle_mod.find_blocks(1, (c[0], c[1]), r, 1.0))


@pytest.mark.parametrize("sort", [False, True])
@pytest.mark.parametrize("slope", [1.0, 0.3, -0.8])
@pytest.mark.parametrize("up", [0.01, 0.9, 2.0, 12.0])
def test_hyperboloid_of_any_size(built, oracle_mod, up, slope, sort):
    clf, cloud = built
    c = cloud.decoded()[cloud.n // 3] + np.array([0.0, 0.0, up if slope > 0 else -up])
    got = clf.points_in(2, c, 0.2, slope, sorted=sort)
    assert np.array_equal(got, oracle_mod.points_in(2, c, 0.2, slope, sorted=sort))


def test_capacity(built):
    from wolkenbase_gb300 import _lib
    clf, cloud = built
    c = cloud.decoded()[cloud.n // 3]
    sh = clf._shape(1, (c[0], c[1]), 1.0, 1.0)
    n = C.c_uint64(0)
    full = clf.points_in(1, (c[0], c[1]), 1.0)
    for cap, want in ((0, _lib.WB_EINVAL), (full.size - 1, _lib.WB_EINVAL), (full.size, 0), (full.size + 5, 0)):
        out = np.full(full.size + 8, 7, np.uint32)
        rc = clf.L.wb_points_in(clf.ctx, C.byref(sh), 0, out.ctypes.data, cap, C.byref(n))
        assert rc == want and n.value == full.size
        assert np.array_equal(out[:full.size], full) if rc == 0 else np.all(out == 7)
        assert np.all(out[full.size:] == 7)


def test_heights_order_the_same_through_a_negative_scale(built):
    # record integers order the heights of the one cloud, the heights themselves
    # those of the other; the points are the same
    import wolkenbase_gb300 as wb
    from wolkenbase_gb300 import synth
    clf, cloud = built
    flipped = synth.Cloud(np.ascontiguousarray(cloud.xyz * np.array([1, 1, -1], np.int32)),
                          (cloud.scale[0], cloud.scale[1], -cloud.scale[2]), cloud.offset, cloud.unit, cloud.minc,
                          cloud.maxc)
    assert np.array_equal(flipped.decoded(), cloud.decoded())
    other = wb.Classifier(0)
    other.build(flipped)
    c = cloud.decoded()[cloud.n // 3]
    for r in (0.3, 2.6, 40.0):
        want = clf.points_in(1, (c[0], c[1]), r, sorted=True)
        assert np.array_equal(other.points_in(1, (c[0], c[1]), r, sorted=True), want)
    other.close()
