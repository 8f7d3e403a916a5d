"""A cloud without records between two runs of another: it reports nothing, and
leaves nothing of itself or of the first to the second.  So does one that is a
context's first."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [0, 4])
def test_empty_cloud_between(cuda_lib_path, shape):
    import wolkenbase_gb300 as wb
    from wolkenbase_gb300 import synth
    cloud = synth.density_tile(6000, 91)
    empty = synth.Cloud(np.zeros((0, 3), np.int32), cloud.scale, cloud.offset, 1.0, cloud.minc, cloud.maxc)
    clf = wb.Classifier(0)
    try:
        clf.set_tuning(shape=shape)
        before = clf.classify_cloud(cloud).copy()
        tiles = clf.tiles().copy()
        assert clf.classify_cloud(empty).size == 0
        info = clf.info()
        assert info["n_points"] == info["n_distinct"] == info["n_leaves"] == 0
        assert not clf.tiles()["n_points"].any() and not clf.tiles()["n_ground"].any()
        assert clf.points_in(1, (0.0, 0.0), 1e6).size == 0 and clf.find_blocks(1, (0.0, 0.0), 1e6).size == 0
        clf.build(empty)
        clf.scan(wb.Params())
        got, margin = clf.classify_margins(wb.Params())
        assert got.size == 0 and margin.size == 0
        assert np.array_equal(clf.classify_cloud(cloud), before)
        assert np.array_equal(clf.tiles(), tiles)
    finally:
        clf.close()


def test_empty_cloud_first(cuda_lib_path):
    import wolkenbase_gb300 as wb
    from wolkenbase_gb300 import synth
    cloud = synth.density_tile(6000, 91)
    empty = synth.Cloud(np.zeros((0, 3), np.int32), cloud.scale, cloud.offset, 1.0, cloud.minc, cloud.maxc)
    clf, other = wb.Classifier(0), wb.Classifier(0)
    try:
        assert clf.classify_cloud(empty).size == 0
        assert clf.tiles().size > 0 and not clf.tiles()["n_points"].any()
        assert np.array_equal(clf.classify_cloud(cloud), other.classify_cloud(cloud))
        assert np.array_equal(clf.tiles(), other.tiles())
    finally:
        clf.close()
        other.close()
