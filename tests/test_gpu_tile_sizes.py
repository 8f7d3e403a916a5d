"""The tile gather and scan over all tile sizes, against the oracle: every tile
figure equal.  The density grows along the cloud, so that tiles of one to more
than 1024 points occur (the gather sorts by powers of two up to 1024, the scan
sums 32 points at a time and keeps 224), over heights with many equal minima, on
slopes, and with a negative record scale."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _cloud(kind, n=60000, seed=7):
    from wolkenbase_gb300 import synth
    r = np.random.default_rng(seed)
    x = 40000 * np.log1p(r.random(n) * 499) / np.log(500)   # density from 1 to 500 along 40 m
    y = r.integers(0, 4000, n)
    z = {"flat": np.zeros(n), "steps": r.integers(0, 3, n) * 700.0, "rough": r.integers(0, 2500, n) * 1.0,
         "steep": 0.8 * y + r.integers(0, 40, n), "negative": r.integers(0, 900, n) - 400.0}[kind]
    xyz = np.stack([x, y, z], 1).astype(np.int32)
    scale = (-0.001, 0.001, 0.001) if kind == "negative" else (0.001, 0.001, 0.001)
    c = synth.Cloud(np.ascontiguousarray(xyz), scale, (0.0, 0.0, 0.0), 1.0, (0, 0, 0), (0, 0, 0))
    d = c.decoded()
    c.minc, c.maxc = tuple(map(float, d.min(axis=0))), tuple(map(float, d.max(axis=0)))
    return c


@pytest.mark.parametrize("kind", ["flat", "steps", "rough", "steep", "negative"])
def test_tiles_of_every_size_match_oracle(classifier, oracle_mod, kind):
    import wolkenbase_gb300 as wb
    cloud = _cloud(kind)
    o = oracle_mod.run(cloud, canonical_order=True, threads=8)["tiles"]
    classifier.build(cloud)
    classifier.scan(wb.Params())
    t = classifier.tiles()
    sizes = t["n_points"]
    for lo, hi in ((1, 32), (33, 64), (65, 128), (129, 224), (225, 256), (257, 512), (513, 1024), (1025, 4096)):
        assert ((sizes >= lo) & (sizes <= hi)).any(), (lo, hi)
    assert np.array_equal(t["ex"], o["ex"]) and np.array_equal(t["ey"], o["ey"])
    for f, of in (("n_points", "n_points"), ("tree_flags", "tree_flags"), ("density", "density"),
                  ("h_scan", "h_scan"), ("hyperboloid_size", "h_final"), ("height", "height")):
        assert np.array_equal(t[f], o[of]), f
