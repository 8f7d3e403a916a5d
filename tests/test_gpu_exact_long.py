"""The exact pass over lists of every length: clouds with a negative scale list
all their points, which blocks of warps take one at a time while they are few and
single warps where they are many, alone and as several jobs of one batch, against
the oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _cloud(n, seed):
    from wolkenbase_gb300 import synth
    r = np.random.default_rng(seed)
    side = max(1.0, 0.07 * n ** 0.5)
    d = np.stack([r.uniform(0, side, n), r.uniform(0, side, n), r.uniform(0, 0.6, n) ** 2], 1)
    d[0], d[-1] = 0.0, (side, side, 0.36)
    scale = (-0.001, 0.001, 0.001)
    c = synth.Cloud(np.rint(d / np.array(scale)).astype(np.int32), scale, (0.0, 0.0, 0.0), 1.0, (0.0,) * 3, (side, side, 0.36))
    return c


@pytest.mark.parametrize("n", [2, 33, 1200, 3600, 3700, 4800, 9000])
def test_one_cloud(classifier, oracle_mod, n):
    import wolkenbase_gb300 as wb
    cloud = _cloud(n, n)
    o = oracle_mod.run(cloud, canonical_order=True, threads=8)
    got = classifier.classify_cloud(cloud, wb.Params())
    bad = np.nonzero((got != o["cls"]) & (o["leaf"] >= 0))[0]
    assert bad.size == 0, f"{bad.size} of {n} labels differ"


@pytest.mark.parametrize("sizes", [(40, 700, 3, 900), (2500, 40, 3000, 1, 1700)])
def test_several_jobs(cuda_lib_path, oracle_mod, sizes):
    import wolkenbase_gb300 as wb
    from wolkenbase_gb300 import _lib
    clouds = [_cloud(n, 100 + n) for n in sizes]
    srv = wb.Server(0, prep_slots=4, flush=_lib.WB_FLUSH_FULL)
    try:
        got = srv.classify_batch(clouds, wb.Params())
    finally:
        srv.close()
    for c, g in zip(clouds, got):
        o = oracle_mod.run(c, canonical_order=True, threads=8)
        assert np.array_equal(np.asarray(g)[o["leaf"] >= 0], o["cls"][o["leaf"] >= 0])
