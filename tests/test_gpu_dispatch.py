"""The forms of a kernel that a launch rule chooses between give identical lanes.

Waves of few lanes run as whole paths, larger ones as the wavefront; rays of deep trees stream
over a warp's lanes after the first event, except in counting runs; evenly spaced knots guess
their segment, others are searched.  Each pair is compared bit for bit, or with the oracle.
"""

import numpy as np
import pytest

from rypath_b200 import abi, renderer, scenes
from tests.oracle_lib import OracleScene, oracle, request
from tests.test_gpu_parity import _soup

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


@pytest.mark.parametrize("width,height,spp", [(257, 129, 1), (200, 170, 3)])
def test_streamed_walks_equal_a_ray_a_thread(width, height, spp):
    rs = build(scenes.mixed_scene(width, height, spp, 16, subdivisions=5, sphere_count=8))
    req = renderer.RenderRequest(width, height, sample_count=spp)
    streamed = rs.sample(req)
    assert streamed.status == abi.RP_SUCCESS, streamed.diagnostic
    rs.set_counting(True)  # counting runs walk a ray a thread
    counted = rs.sample(req)
    rs.set_counting(False)
    assert_same(streamed.packet_samples, counted.packet_samples)
    rs.close()


@pytest.mark.parametrize("spp", [4736, 4737])
def test_scalar_waves_at_the_slot_count(spp):
    # 64 lanes a sample: as many lanes as the slots of 148 SMs, then more, the last ones in slots
    # that others left
    rs = build(scenes.cornell_fog(8, 8, 1, 8))
    whole = rs.sample_scalar(renderer.RenderRequest(8, 8, sample_count=spp)).samples
    part = rs.sample_scalar(renderer.RenderRequest(8, 8, sample_begin=spp - 1, sample_count=1)).samples
    assert whole.tobytes()[-part.nbytes:] == part.tobytes()
    rs.close()


def uneven(scene, kind):
    """The scene with its sampled spectra on two knots, on uneven ones, or inside the visible range
    (the values outside are zero, or the ends' for optical constants)."""
    w = {"two": [360.0, 830.0], "uneven": [360.0, 365.0, 400.0, 612.5, 613.0, 830.0],
         "inside": [420.0, 500.0, 580.0, 660.0]}[kind]
    knots, ranges = [], {}
    old = np.asarray(scene.knots)

    def moved(begin, count):
        if count < 2:
            return begin, count
        if begin not in ranges:
            k = old[begin:begin + count]
            ranges[begin] = sum(len(x) for x in knots)
            knots.append(np.stack([np.float32(w), np.interp(w, k[:, 0], k[:, 1]).astype(np.float32)], 1))
        return ranges[begin], len(w)

    for m in scene.materials:
        m.knot_begin, m.knot_count = moved(m.knot_begin, m.knot_count)
        m.eta_begin, m.eta_count = moved(m.eta_begin, m.eta_count)
        m.k_begin, m.k_count = moved(m.k_begin, m.k_count)
    scene.knots = np.concatenate(knots).astype(np.float32)
    return scene


@pytest.mark.parametrize("kind", ["two", "uneven", "inside"])
@pytest.mark.parametrize("transport", [abi.TRANSPORT_HERO, abi.TRANSPORT_SCALAR])
def test_sampled_spectra_on_other_knots(kind, transport):
    scene = uneven(scenes.cornell_microfacets(32, 32, 4, 8, transport=transport), kind)
    rs, ref_scene, q = build(scene), OracleScene(scene), request(32, 32, 4)
    if transport == abi.TRANSPORT_HERO:
        got, ref = rs.sample(renderer.RenderRequest(32, 32, sample_count=4)).packet_samples, ref_scene.sample(q)
    else:
        got, ref = rs.sample_scalar(renderer.RenderRequest(32, 32, sample_count=4)).samples, ref_scene.sample_scalar(q)
    np.testing.assert_array_equal(got["status"], ref["status"])
    # the lane gate of the transports' parity tests: relative 1e-3 for at least 97% of the lanes
    g, r = got["radiance"].reshape(len(got), -1), ref["radiance"].reshape(len(ref), -1)
    close = np.all(np.abs(g - r) <= 1e-3 * np.maximum(np.abs(r), 1e-6) + 1e-7, axis=1)
    assert close.mean() >= 0.97
    rs.close()


@pytest.mark.parametrize("transport", [abi.TRANSPORT_HERO, abi.TRANSPORT_SCALAR])
@pytest.mark.parametrize("limit", [1, 4096])
def test_failed_lanes_are_reported(transport, limit):
    # two panes in a row: camera rays through both exceed a limit of one crossing
    scene = scenes.cornell_pass_through(16, 16, 2, 8, invisible_light=False, mixes=False)
    scene.transport = transport
    second = scenes.identity_instance(scene.positions.shape[0], scene.triangles.shape[0], 2,
                                      scene.instances[-1].material)
    scene.positions = np.concatenate([scene.positions, scene.positions[-4:] + np.float32([0, 0, 0.1])])
    scene.triangles = np.concatenate([scene.triangles, scene.triangles[-2:]])
    scene.instances.append(second)
    rs = build(scene)

    def sample(**more):
        req = renderer.RenderRequest(16, 16, sample_count=2, boundary_limit=limit, **more)
        if transport == abi.TRANSPORT_HERO:
            res = rs.sample(req)
            return res, res.packet_samples
        res = rs.sample_scalar(req)
        return res, res.samples

    res, lanes = sample()
    failed = np.flatnonzero(lanes["status"])
    assert (len(failed) > 0) == (limit == 1)
    assert res.status == (abi.RP_FAILURE if len(failed) else abi.RP_SUCCESS)
    if len(failed):
        assert res.diagnostic.endswith(f"failed with status {lanes['status'][failed[0]]} at lane {failed[0]}")
    refused, lanes = sample(pixel_begin=1, pixel_count=256)
    assert refused.status == abi.RP_INVALID_ARGUMENT and not lanes.tobytes().strip(b"\0")
    rs.close()


@pytest.mark.parametrize("subdivisions", [1, 5])  # a tree whose scalar walks pair, one whose walks stream
def test_scalar_walks_match_the_oracle(subdivisions):
    scene = scenes.mixed_scene(32, 32, 4, 8, subdivisions=subdivisions, sphere_count=3)
    scene.transport = abi.TRANSPORT_SCALAR
    rs = build(scene)
    got = rs.sample_scalar(renderer.RenderRequest(32, 32, sample_count=4)).samples
    ref = OracleScene(scene).sample_scalar(request(32, 32, 4))
    np.testing.assert_array_equal(got["status"], ref["status"])
    close = np.abs(got["radiance"] - ref["radiance"]) <= 1e-3 * np.maximum(np.abs(ref["radiance"]), 1e-6) + 1e-7
    assert close.mean() >= 0.97
    rs.close()


@pytest.mark.parametrize("n", [2, 2049, 131072, 131073, 270001])  # tiles of 2,048, scan passes of 64 tiles
def test_sorted_order_is_the_oracles(n):
    scene = _soup(n, 9)
    rs, oracle_scene = build(scene), OracleScene(scene)
    nodes, order, keys, bounds = rs.export_bvh(n)
    rs.close()
    ref = [np.zeros((n - 1, 3), np.uint32), np.zeros(n, np.uint32), np.zeros(n, np.uint64),
           np.zeros((2 * n - 1, 6), np.float32)]
    assert oracle().or_export_bvh(oracle_scene.handle, *(a.ctypes.data for a in ref), n) == n
    np.testing.assert_array_equal(keys, ref[2])
    np.testing.assert_array_equal(order, ref[1])


@pytest.mark.parametrize("subdivisions", [1, 3, 5])
def test_scalar_walks_of_deep_trees_take_one_trip_an_event(subdivisions):
    # without media a walk takes a path's connection together with its next ray: at most depth + 2
    # trips of a walk and a step, in eights, beside the camera rays, the slots' two kernels, the draw
    # tables and the lanes
    scene = scenes.mixed_scene(128, 128, 1, 6, subdivisions=subdivisions, sphere_count=8)
    scene.transport = abi.TRANSPORT_SCALAR
    rs = build(scene)
    assert rs.sample_scalar(renderer.RenderRequest(128, 128)).status == abi.RP_SUCCESS
    assert rs.timing().kernel_launches <= 2 * 8 + 5
    rs.close()


@pytest.mark.parametrize("kind,limit", [("point", 18432), ("texture", 18432), ("cauchy", 4608), ("mixed", 8704)])
def test_the_form_that_a_wave_takes(kind, limit):
    # the pairs compared above are of two forms: whole paths launch no closest-hit kernel of their own
    rs = build(small_scene(kind, 257, 129))
    for count, wavefront in ((1, False), (limit, False), (limit + 1, True), (257 * 129, True)):
        assert rs.sample(renderer.RenderRequest(257, 129, pixel_count=count)).status == abi.RP_SUCCESS
        assert (rs.timing().trace_launches > 0) == wavefront
    rs.close()


@pytest.mark.parametrize("depth,limit", [(3, 64), (15, 64), (19, 2048)])  # 512 lanes an event past the sixteenth, 64
def test_closed_scenes_with_rough_dielectrics_take_the_wavefront_earlier(depth, limit):
    rs = build(scenes.cornell_microfacets(64, 64, 1, depth, transport=abi.TRANSPORT_HERO))
    whole = rs.sample(renderer.RenderRequest(64, 64))
    assert whole.status == abi.RP_SUCCESS, whole.diagnostic
    assert rs.timing().trace_launches > 0
    for begin, count in ((0, 1), (1500, limit), (1500, limit + 1)):
        part = rs.sample(renderer.RenderRequest(64, 64, pixel_begin=begin, pixel_count=count))
        assert part.status == abi.RP_SUCCESS, part.diagnostic
        assert (rs.timing().trace_launches > 0) == (count > limit)
        assert_same(part.packet_samples, whole.packet_samples[begin:begin + count])
    rs.close()


@pytest.mark.parametrize("kind", ["fog", "shallow", "deep"])
def test_scalar_lanes_in_refilled_slots(kind):
    # more lanes than the wave's slots (2,048 an SM): every lane once, as in waves that fill them once
    torch = pytest.importorskip("torch")
    slots = 2048 * torch.cuda.get_device_properties(0).multi_processor_count
    if kind == "fog":
        scene = scenes.cornell_fog(64, 64, 1, 8)
    else:
        scene = scenes.mixed_scene(64, 64, 1, 8, subdivisions=1 if kind == "shallow" else 5, sphere_count=4)
        scene.transport = abi.TRANSPORT_SCALAR
    rs = build(scene)
    for spp in (slots // 4096, slots // 4096 + 1, slots // 4096 + 17):
        whole = rs.sample_scalar(renderer.RenderRequest(64, 64, sample_count=spp)).samples
        half = spp // 2
        parts = [rs.sample_scalar(renderer.RenderRequest(64, 64, sample_begin=b, sample_count=n)).samples
                 for b, n in ((0, half), (half, spp - half))]
        assert whole.tobytes() == np.concatenate(parts).tobytes()
    rs.close()


@pytest.mark.parametrize("transport", [abi.TRANSPORT_HERO, abi.TRANSPORT_SCALAR])
@pytest.mark.parametrize("lanes", [1, 1024, 1025])  # the most whose statuses the host reads, and one more
def test_the_first_failed_lane_is_reported(transport, lanes):
    # a boundary limit of one crossing, and two panes in a row before part of the film
    scene = scenes.cornell_pass_through(64, 64, 1, 8, invisible_light=False, mixes=False)
    scene.transport = transport
    second = scenes.identity_instance(scene.positions.shape[0], scene.triangles.shape[0], 2,
                                      scene.instances[-1].material)
    scene.positions = np.concatenate([scene.positions, scene.positions[-4:] + np.float32([0, 0, 0.1])])
    scene.triangles = np.concatenate([scene.triangles, scene.triangles[-2:]])
    scene.instances.append(second)
    rs = build(scene)
    sample = rs.sample if transport == abi.TRANSPORT_HERO else rs.sample_scalar

    def run(begin):
        res = sample(renderer.RenderRequest(64, 64, pixel_begin=begin, pixel_count=lanes, boundary_limit=1))
        return res, (res.samples if transport == abi.TRANSPORT_SCALAR else res.packet_samples)["status"]

    whole = sample(renderer.RenderRequest(64, 64, boundary_limit=1))
    status = (whole.samples if transport == abi.TRANSPORT_SCALAR else whole.packet_samples)["status"]
    first = int(np.flatnonzero(status)[0])
    for begin in (first, max(0, first - lanes + 1), int(np.flatnonzero(status == 0)[0])):
        res, got = run(begin)
        np.testing.assert_array_equal(got, status[begin:begin + lanes])
        failed = np.flatnonzero(got)
        assert res.status == (abi.RP_FAILURE if len(failed) else abi.RP_SUCCESS)
        if len(failed):
            assert res.diagnostic.endswith(f"failed with status {got[failed[0]]} at lane {failed[0]}")
    rs.close()
