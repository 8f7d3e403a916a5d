"""A thickness tens of thousands of times the hyperboloid's polar radius, against the
oracle: points of a plane two kilometres above another one, whose hyperboloids end
a few parts in a thousand of a polar radius below the lower plane.  The FP32 values
of such a centre are off by more than that; whether a box is read must not depend
on it.  The parameters are those, of millions drawn, at which the rounding of the
envelope's apex (the first two) and of the height differences (the others) is
worst."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# scale, distance of the planes and spacing of the lower one in record units, the parameters
CASES = {"reach_63mm": (0.001, 2302122, 14, dict(max_slope=0.02922, min_hyp_size=31.075, thickness=2302.121942)),
         "reach_125mm": (0.001, 2302122, 24, dict(max_slope=0.01461, min_hyp_size=134.182, thickness=2302.121942)),
         "reach_280mm": (0.01, 100001, 8, dict(max_slope=0.004, min_hyp_size=1562.437, thickness=1000.009975)),
         "reach_1120mm": (0.01, 200003, 14, dict(max_slope=0.004, min_hyp_size=6250.083, thickness=2000.0299))}


def _cloud(scale, distance, spacing, seed=1, m=60):
    from wolkenbase_gb300 import synth
    r = np.random.default_rng(seed)
    low = np.stack(np.meshgrid(np.arange(m) * spacing, np.arange(m) * spacing), -1).reshape(-1, 2)
    low = low + r.integers(-3, 4, low.shape)
    high = r.integers(10 * spacing, (m - 10) * spacing, (120, 2))
    xyz = np.concatenate([np.c_[low, np.zeros(len(low), int)], np.c_[high, np.full(len(high), distance)]])
    c = synth.Cloud(np.ascontiguousarray(xyz[r.permutation(len(xyz))], np.int32), (scale,) * 3, (0.0,) * 3, 1.0,
                    (0, 0, 0), (0, 0, 0))
    d = c.decoded()
    c.minc, c.maxc = tuple(map(float, d.min(axis=0))), tuple(map(float, d.max(axis=0)))
    return c


@pytest.mark.parametrize("kernel", ["groups", "points", "bins"])
@pytest.mark.parametrize("name", sorted(CASES))
def test_labels(classifier, oracle_mod, name, kernel):
    import wolkenbase_gb300 as wb
    scale, distance, spacing, p = CASES[name]
    cloud = _cloud(scale, distance, spacing)
    p = dict(p, tile_size=1000.0)
    o = oracle_mod.run(cloud, canonical_order=True, threads=8, **p)
    high = cloud.xyz[:, 2] > 0
    assert np.mean(o["cls"][high] == 1) > 0.8
    keep = classifier.tuning()
    classifier.set_tuning(shape=4 if kernel == "points" else 0)
    try:
        classifier.build(cloud)
        classifier.scan(wb.Params(**p))
        got = classifier.classify_margins(wb.Params(**p))[0] if kernel == "bins" else classifier.classify(wb.Params(**p))
    finally:
        classifier.set_tuning(shape=keep["shape"])
    bad = np.nonzero((got != o["cls"]) & (o["leaf"] >= 0))[0]
    assert bad.size == 0, f"{bad.size} labels differ, {np.sum(high[bad])} of them of high points"
