"""Calls that want margins work on column groups of the grid: formed by the first
such call, kept while the grid stands, formed again for the next cloud; a call
without margins in between changes nothing."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _launched(clf, call):
    before = clf.launch_count()
    out = call()
    return clf.launch_count() - before, out


def test_column_groups_are_formed_once_per_grid(cuda_lib_path):
    import wolkenbase_gb300 as wb
    from wolkenbase_gb300 import synth
    clf = wb.Classifier(0)
    try:
        for seed in (92, 93):
            cloud = synth.density_tile(9000 + seed, seed)
            clf.build(cloud)
            clf.scan(wb.Params())
            first, a = _launched(clf, lambda: clf.classify_margins(wb.Params()))
            again, b = _launched(clf, lambda: clf.classify_margins(wb.Params()))
            assert first - again == 3   # counted, summed up and filled
            cls = clf.classify(wb.Params())
            third, c = _launched(clf, lambda: clf.classify_margins(wb.Params()))
            assert third == again
            for got in (b, c):
                assert np.array_equal(got[0], a[0]) and np.array_equal(got[1], a[1], equal_nan=True)
            assert np.array_equal(cls, a[0])
    finally:
        clf.close()
