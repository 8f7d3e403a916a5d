"""The exact pass, a block of warps per point: high points whose widest gap is 144
degrees to within the rounding of their neighbours' places, with none to thousands
of further neighbours on the other side, against the oracle; some end ground, some
not."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _cloud(fill, seed):
    from wolkenbase_gb300 import synth
    r = np.random.default_rng(seed)
    pts = []
    for k in range(6):
        cx, cy = 400_000 * (k % 3), 400_000 * (k // 3)
        pts.append((cx, cy, 150_000))
        theta = r.random() * 2 * np.pi
        ang = theta + np.radians([0.0, 144.0, 252.0])
        rad = r.uniform(5e4, 1e5, 3)
        # the rest lies between the second and the first direction, away from the gap
        ang = np.concatenate([ang, theta + np.radians(r.uniform(146.0, 358.0, fill))])
        rad = np.concatenate([rad, r.uniform(2e3, 1e5, fill)])
        pts += list(zip(cx + rad * np.cos(ang), cy + rad * np.sin(ang), r.integers(0, 2000, len(ang))))
    xyz = np.rint(np.array(pts)).astype(np.int32)
    c = synth.Cloud(np.ascontiguousarray(xyz), (0.001, 0.001, 0.001), (0.0, 0.0, 0.0), 1.0, (0, 0, 0), (0, 0, 0))
    d = c.decoded()
    c.minc, c.maxc = tuple(map(float, d.min(axis=0))), tuple(map(float, d.max(axis=0)))
    return c


@pytest.mark.parametrize("fill", [0, 3, 40, 700])
@pytest.mark.parametrize("seed", [1, 2])
def test_gaps_of_144_degrees(classifier, oracle_mod, fill, seed):
    import wolkenbase_gb300 as wb
    cloud = _cloud(fill, seed)
    p = wb.Params(tile_size=50.0)
    o = oracle_mod.run(cloud, canonical_order=True, threads=8, tile_size=50.0)
    classifier.build(cloud)
    classifier.scan(p)
    got = classifier.classify(p)
    assert np.array_equal(got, o["cls"])
    _, margin = classifier.classify_margins(p)
    assert (np.abs(margin[::4 + fill]) < 5e-4).any()   # degrees: within the fast pass's doubt
