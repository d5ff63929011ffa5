"""Ray queries at the edges of the box test's arithmetic, bit for bit against a scan of every triangle.

Axis-parallel directions with zeros of either sign, components so small that their reciprocal
or whose product with a distance overflows, very long and very short directions, origins on box
planes and far outside, and limits at, before and behind the hit.
"""

import numpy as np
import pytest

from rypath_b200 import abi, renderer, scenes
from tests.oracle_lib import OracleScene, oracle
from tests.test_gpu_parity import _soup

pytestmark = pytest.mark.gpu


def _axis(rng, n):
    """Directions along an axis, with zeros of either sign, or in an axis plane."""
    d = rng.choice(np.array([0.0, -0.0, 1.0, -1.0, 0.5]), (n, 3))
    d[np.arange(n), rng.integers(0, 3, n)] = rng.choice([1.0, -1.0], n)
    return d


def _directions(kind, rng, n):
    if kind == "axis":
        return _axis(rng, n)
    d = rng.normal(size=(n, 3))
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    if kind == "tiny":  # one or two components whose reciprocal is huge or overflows
        k = rng.integers(0, 3, n)
        for c in range(2):
            use = rng.random(n) < (1.0 if c == 0 else 0.5)
            v = rng.choice([1.0, -1.0], n) * 10.0 ** rng.uniform(-45, -20, n)
            d[np.flatnonzero(use), ((k + c) % 3)[use]] = v[use]
    elif kind == "scaled":
        d *= 10.0 ** rng.uniform(-25, 25, (n, 1))
    return d


def _rays(scene, kind, n, seed):
    rng = np.random.default_rng(seed)
    lo, hi = scene.positions.min(0).astype(np.float64), scene.positions.max(0).astype(np.float64)
    d = _directions(kind, rng, n)
    o = rng.uniform(lo, hi, (n, 3))
    third = n // 3
    # on the planes of triangles' boxes: some or all coordinates of a vertex
    v = scene.positions[rng.integers(0, len(scene.positions), third)]
    o[:third] = np.where(rng.random((third, 3)) < 0.6, v, o[:third])
    # outside, aimed at a point inside: a few scene sizes away, or a thousand
    far = (hi - lo).max() * 10.0 ** rng.uniform(0, 3, (third, 1))
    unit = d[third:2 * third] / np.abs(d[third:2 * third]).max(1, keepdims=True)
    o[third:2 * third] -= far * unit
    return np.concatenate([o, d, np.full((n, 1), np.inf)], 1).astype(np.float32)


def _scan(scene, rays):
    hits = np.zeros((len(rays), 4), np.float32)
    handle = OracleScene(scene)
    oracle().or_trace_rays(handle.handle, rays.ctypes.data, len(rays), 0, 1, hits.ctypes.data)
    return hits


@pytest.mark.parametrize("kind", ["axis", "tiny", "scaled"])
@pytest.mark.parametrize("model", ["cornell", "soup", "sheet"])
def test_ray_queries_match_a_scan(model, kind):
    scene = {"cornell": lambda: scenes.cornell_box(8, 8, 1), "soup": lambda: _soup(3000, 3),
             "sheet": lambda: _soup(3000, 4)}[model]()
    if model == "sheet":  # every box is flat
        scene.positions[:, 1] = np.float32(0.25)
    built = renderer.build_renderer(scene)
    assert built.status == abi.RP_SUCCESS, built.diagnostic
    rs = built.scene
    rays = _rays(scene, kind, 12000, 7)
    ref = _scan(scene, rays)
    hit = ref[:, 3].view(np.uint32) != abi.RP_NONE
    assert hit.sum() > (100 if model != "sheet" else 10)
    # the same rays ending at the hit, one step before it and some way behind it (the hit's own
    # rounding, of about 2^-24 of the distances that went into it, is not the box test's)
    limited = np.repeat(rays[hit], 3, axis=0)
    t, size = ref[hit, 0], (scene.positions.max(0) - scene.positions.min(0)).max()
    limited[0::3, 6], limited[1::3, 6] = t, np.nextafter(t, np.float32(0))
    limited[2::3, 6] = t + np.float32(1e-3) * (t + size / np.abs(rays[hit, 3:6]).max(1))
    for r, expected in ((rays, ref), (limited, _scan(scene, limited))):
        got = rs.trace(r)
        np.testing.assert_array_equal(got.view(np.uint32), expected.view(np.uint32))
        any_hit = rs.trace(r, any_hit=True)
        np.testing.assert_array_equal(any_hit[:, 0] == 1, expected[:, 3].view(np.uint32) != abi.RP_NONE)
    rs.close()
