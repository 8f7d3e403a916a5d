"""A look-back wait that runs out: the waiting block returns without writing, every
call whose scan or sort gave up answers WB_ETIMEDOUT and clears the context's
error word, and the next call gives the right result again.  The waits run out in
kernels with a short limit (a status word that nothing publishes); in whole calls
the error word is set beforehand, which is what their kernels find after one."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def shim(cuda_lib_path, tmp_path_factory):
    from wolkenbase_gb300 import _build
    out = str(tmp_path_factory.mktemp("shim") / "shim.so")
    cmd = [_build.nvcc()] + _build._flags("shim.cu") + ["-DWB_LOOKBACK_SPINS=2000", "-shared", "-o", out,
                                                       os.path.join(ROOT, "tests", "lookback_shim.cu"), cuda_lib_path]
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    L = C.CDLL(out)
    for f in ("shim_set", "shim_get", "shim_grid"):
        getattr(L, f).argtypes = [C.c_void_p] + {"shim_set": [C.c_int], "shim_get": [C.c_void_p], "shim_grid": []}[f]
    return L


@pytest.mark.parametrize("n", [256, 257, 5000])
@pytest.mark.parametrize("first", [0, 1])
def test_scan_gives_up(shim, n, first):
    out, total, err = np.zeros(n, np.uint32), C.c_uint32(0), C.c_int(0)
    assert shim.shim_scan(n, first, out.ctypes.data_as(C.c_void_p), C.byref(total), C.byref(err)) == 0
    if first == 0:
        assert err.value == 0 and total.value == n and np.array_equal(out, np.arange(n))
    else:
        assert (err.value == 1) == (n > 256) and total.value == 7 and np.all(out == 7)


@pytest.mark.parametrize("there", [0, 1, 2, 3])
def test_column_gives_up(shim, there):
    """Tile 2 is the nearest: unpublished, it is waited for in vain."""
    gave, err = C.c_int(0), C.c_int(0)
    assert shim.shim_column(there, C.byref(gave), C.byref(err)) == 0
    assert (gave.value, err.value) == ((0, 0) if there == 3 else (32, 1))


def _cloud(n=20000):
    from wolkenbase_gb300 import synth
    return synth.density_tile(n, 83)


def _calls():
    import wolkenbase_gb300 as wb
    from wolkenbase_gb300 import _lib
    whole = (_lib.WB_SHAPE_CYLINDER, (5.0, 5.0), 1e6)

    def scan(clf, size):
        clf.scan(wb.Params(tile_size=size))
        return clf.tiles().copy()

    def margins(clf):
        clf.scan(wb.Params())
        return clf.classify_margins(wb.Params())[0]

    def split(clf, stride):
        rec = np.random.default_rng(5).integers(0, 32, (3000, stride)).astype(np.uint8)
        return np.concatenate([np.asarray(x).ravel() for x in clf.las_split_by_class(rec, 1 if stride == 28 else 6)])

    return {
        "build": lambda clf: (clf.build(_cloud()), clf.store_order())[1],
        "scan": lambda clf: scan(clf, 1.0),
        "scan_large_tiles": lambda clf: scan(clf, 20.0),
        "find_blocks": lambda clf: clf.find_blocks(*whole),
        "points_in_few": lambda clf: clf.points_in(_lib.WB_SHAPE_CYLINDER, (5.0, 5.0), 0.5, sorted=True),
        "points_in_many": lambda clf: clf.points_in(*whole, sorted=True),
        "split_words": lambda clf: split(clf, 28),
        "split_bytes": lambda clf: split(clf, 30),
    }


@pytest.mark.parametrize("name", ["build", "scan", "scan_large_tiles", "find_blocks", "points_in_few", "points_in_many",
                                  "split_words", "split_bytes"])
def test_call_answers_timed_out(shim, cuda_lib_path, name):
    import wolkenbase_gb300 as wb
    from wolkenbase_gb300 import _lib
    call = _calls()[name]
    clf = wb.Classifier(0)
    try:
        clf.build(_cloud())
        want = call(clf)
        assert shim.shim_set(clf.ctx, 1) == 0
        with pytest.raises(wb.WolkenbaseError) as e:
            call(clf)
        assert e.value.code == _lib.WB_ETIMEDOUT, str(e.value)
        word = C.c_int(5)
        assert shim.shim_get(clf.ctx, C.byref(word)) == 0 and word.value == 0
        assert np.array_equal(call(clf), want)
    finally:
        clf.close()


def test_grid_and_column_groups_answer_timed_out(shim, cuda_lib_path):
    import wolkenbase_gb300 as wb
    from wolkenbase_gb300 import _lib
    clf = wb.Classifier(0)
    try:
        cloud = _cloud()
        want = clf.classify_cloud(cloud)
        assert shim.shim_set(clf.ctx, 1) == 0
        assert shim.shim_grid(clf.ctx) == _lib.WB_ETIMEDOUT
        assert shim.shim_grid(clf.ctx) == 0
        clf.scan(wb.Params())
        assert np.array_equal(clf.classify(wb.Params()), want)
        assert shim.shim_set(clf.ctx, 1) == 0
        with pytest.raises(wb.WolkenbaseError) as e:
            clf.classify_margins(wb.Params())
        assert e.value.code == _lib.WB_ETIMEDOUT
        assert np.array_equal(clf.classify_margins(wb.Params())[0], want)
    finally:
        clf.close()
