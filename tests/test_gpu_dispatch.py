"""The forms of a kernel that a launch rule chooses between give identical lanes.

Waves of few lanes run as whole paths, larger ones as the wavefront, compared bit for bit.
"""

import numpy as np
import pytest

from rypath_b200 import abi, renderer, scenes

pytestmark = pytest.mark.gpu

FIELDS = ("status", "pixel", "sample_low", "sample_high", "wavelengths", "wavelength_pdfs", "radiance")


def build(scene):
    built = renderer.build_renderer(scene)
    assert built.status == abi.RP_SUCCESS, built.diagnostic
    return built.scene


def assert_same(a, b):
    for f in FIELDS:
        np.testing.assert_array_equal(a[f], b[f], err_msg=f)


def small_scene(kind, width, height):
    if kind == "mixed":
        return scenes.mixed_scene(width, height, 1, 16, subdivisions=3, sphere_count=8)
    if kind == "sky":
        return scenes.with_environment_image(scenes.mixed_scene(width, height, 1, 6, subdivisions=2, sphere_count=4),
                                             width=32)
    return scenes.cornell_features(kind, width, height, 1, 8)


# the largest wave that runs as whole paths: 512 lanes an event (max depth + 1 of them), 2,048 in
# scenes of one BSDF family
@pytest.mark.parametrize("kind,limit", [("point", 18432), ("texture", 18432), ("cauchy", 4608), ("mixed", 8704),
                                        ("sky", 3584)])
@pytest.mark.parametrize("sampler", [abi.SAMPLER_SOBOL, abi.SAMPLER_INDEPENDENT])
def test_whole_paths_equal_the_wavefront(kind, limit, sampler):
    rs = build(small_scene(kind, 257, 129))  # 33,153 lanes: a wavefront
    whole = rs.sample(renderer.RenderRequest(257, 129, sampler=sampler))
    assert whole.status == abi.RP_SUCCESS, whole.diagnostic
    for begin, count in ((0, limit), (31, 1), (5000, 63), (129, 65), (7, limit + 1)):
        part = rs.sample(renderer.RenderRequest(257, 129, sampler=sampler, pixel_begin=begin, pixel_count=count))
        assert part.status == abi.RP_SUCCESS, part.diagnostic
        assert_same(part.packet_samples, whole.packet_samples[begin:begin + count])
    rs.close()
