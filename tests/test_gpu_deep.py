"""Trees as deep as the traversal stacks and deeper: every form of the walks gives the same lanes.

Nested groups of triangles on a line of Morton cells that halves every third group, each group's
boxes larger than those of all later groups together: every wide node holds one group and the
node of the rest, so a scene of g groups has g + 1 wide levels, and a ray through the middle
leaves a group behind on the stack at each of them.  Trees of at most 16 levels walk with the
short stack, deeper ones with 40 entries; a query that needs more fails (status 3).
"""

import numpy as np
import pytest

from rypath_b200 import abi, renderer, scenes
from tests.oracle_lib import OracleScene, request

pytestmark = pytest.mark.gpu

STACK = 40


def deep_scene(groups, width, height):
    """A floor under the groups, slivers along their boxes' diagonals (few rays meet them) but for
    group 40's: standing triangles, which shadow the floor from the light on its other side."""
    sliver = np.array([(-1, -1, -1), (1, 1, 1), (1, 1, 1 - 2.0 ** -12)])
    triangles = []
    for g in range(groups):
        centre = np.zeros(3)
        centre[g % 3] = 2.0 ** -(g // 3 + 1)
        half = np.round((0.25 + 4 * 2.0 ** (-g / 3) + (63 - g) / 256) * 2 ** 18) / 2 ** 18
        shape = np.array([(-1, -1, -1), (1, 1, -1), (0, 0, 1)]) if g == STACK else sliver
        triangles += [centre + half * shape] * 16
    triangles += [0.25 * sliver] * 2 + [1 + 4.5 * sliver] * 2  # the cells' corners (0, 0, 0) and (1, 1, 1)
    a, b, c, d = np.array([(-24, -24, 0), (24, -24, 0), (24, 24, 0), (-24, 24, 0)]) + [0.5, 0, 0]
    triangles += [np.stack([a, b, c]), np.stack([a, c, d])]
    s = scenes.cornell_box(width, height, 1, 3)
    s.positions = np.concatenate(triangles).astype(np.float32)
    n = len(triangles)
    s.triangles = np.arange(3 * n, dtype=np.uint32).reshape(-1, 3)
    s.instances = [scenes.identity_instance(0, 0, n, 0)]
    s.emissions = []
    s.positional = [{"kind": abi.POINT_LIGHT, "position": (14.0, 0.1, 0.1),
                     "intensity": scenes.blackbody_emission(5000, 900.0)}]
    s.camera = scenes.pinhole_camera((-12, 0, 6), (-12, 0, 0), (0, 1, 0), 20.0, width, height)
    return s


def wide_levels(rs, n):
    nodes, _ = rs.export_wide(n)
    inner = nodes[:, 15]
    base = np.ascontiguousarray(nodes[:, 16:20]).view(np.uint32)[:, 0]
    levels, level = 0, [0]
    while level:
        levels += 1
        level = [int(base[i]) + k for i in level for k in range(bin(inner[i]).count("1"))]
    return levels


# the last tree of the short stack, the first of the deep one, the deepest that it holds, the
# first beyond it and one whose shadow rays through the middle need more than it
@pytest.mark.parametrize("groups", [15, 16, 39, 40, 62])
def test_walks_of_deep_trees_agree(groups):
    width = height = 96  # 9,216 lanes: a wavefront at depth 3, whole paths in parts
    scene = deep_scene(groups, width, height)
    built = renderer.build_renderer(scene)
    assert built.status == abi.RP_SUCCESS, built.diagnostic
    rs = built.scene
    assert wide_levels(rs, scene.triangle_count) == groups + 1
    req = renderer.RenderRequest(width, height)
    plain = rs.sample(req).packet_samples
    assert rs.timing().trace_launches == 4
    rs.set_counting(True)  # counting runs walk a ray a thread
    counted = rs.sample(req).packet_samples
    rs.set_counting(False)
    parts = []
    for begin in range(0, width * height, 3072):
        parts.append(rs.sample(renderer.RenderRequest(width, height, pixel_begin=begin, pixel_count=3072)).packet_samples)
        assert rs.timing().trace_launches == 0
    parts = np.concatenate(parts)
    rs.close()
    for f in ("status", "pixel", "wavelengths", "wavelength_pdfs", "radiance"):
        np.testing.assert_array_equal(plain[f], counted[f], err_msg=f)
        np.testing.assert_array_equal(plain[f], parts[f], err_msg=f)
    ok = plain["status"] == 0
    assert ok.all() if groups < STACK else set(np.unique(plain["status"])) <= {0, 3}
    assert groups < 62 or not ok.all()
    ref = OracleScene(scene).sample(request(width, height, 1))
    # the lane gate of the transports' parity tests: relative 1e-3 for at least 97% of the lanes
    close = np.all(np.abs(plain["radiance"] - ref["radiance"]) <= 1e-3 * np.maximum(np.abs(ref["radiance"]), 1e-6) + 1e-7,
                   axis=1)
    assert close[ok].mean() >= 0.97
