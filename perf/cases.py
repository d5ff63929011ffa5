"""Performance cases of the renderer: what a program that uses it has it do.

Every case goes through the public Python entry points (rypath_b200.renderer): a frame session's
frame, a packet request to host memory, film renders of both transports into a device film, a
batch of views, a whole progressive job from host arrays to a host film, closest-hit queries and
an adjoint gradient.  Scene generators, sizes and sample counts are those of the package's own
benchmark and tests, with ragged films and other samplers among them.

A state's scene is resident (built once, as a program that renders more than one image keeps it)
except in the progressive job, whose pass builds it.
"""

import math

import numpy as np
import torch

from rypath_b200 import abi, renderer, scenes

FILM_DOUBLES = abi.FILM_PIXEL_BYTES // 8
SAMPLERS = {"independent": abi.SAMPLER_INDEPENDENT, "sobol": abi.SAMPLER_SOBOL, "halton": abi.SAMPLER_HALTON,
            "zsobol": abi.SAMPLER_ZSOBOL}

# Scenes by name: (generator of (case, seed), triangles, rays per sample, events per sample).
# The mixed-material scene takes its geometry and materials from the seed; the Cornell-style
# boxes are fixed models, and their renders take the sampler's seed from it.
SCENES = {
    "cornell": (lambda c, s: scenes.cornell_box(c["width"], c["height"], c["spp"], c["depth"]), 36, 8.0, 4.5),
    "cauchy": (lambda c, s: scenes.cornell_features("cauchy", c["width"], c["height"], c["spp"], c["depth"]), 36, 8.0, 4.5),
    "texture": (lambda c, s: scenes.cornell_features("texture", c["width"], c["height"], c["spp"], c["depth"]), 36, 8.0, 4.5),
    "point": (lambda c, s: scenes.cornell_features("point", c["width"], c["height"], c["spp"], c["depth"]), 36, 8.0, 4.5),
    "pass_through": (lambda c, s: scenes.cornell_pass_through(c["width"], c["height"], c["spp"], c["depth"]), 40, 8.0, 4.5),
    "groups": (lambda c, s: scenes.cornell_groups(c["width"], c["height"], c["spp"], c["depth"])[0], 36, 8.0, 4.5),
    "fog": (lambda c, s: scenes.cornell_fog(c["width"], c["height"], c["spp"], c["depth"]), 38, 8.3, 4.5),
    "microfacets": (lambda c, s: scenes.cornell_microfacets(c["width"], c["height"], c["spp"], c["depth"]), 36, 8.0, 4.5),
    "demo": (lambda c, s: scenes.demo_scene(c["width"], c["height"], c["spp"], c["depth"]), 26, 4.0, 2.5),
    "mixed": (lambda c, s: scenes.mixed_scene(c["width"], c["height"], c["spp"], c["depth"], seed=1 + s % 997,
                                              subdivisions=c["subdivisions"], sphere_count=c["spheres"]), 0, 2.3, 1.5),
    "mixed_sky": (lambda c, s: scenes.with_environment_image(
        scenes.mixed_scene(c["width"], c["height"], c["spp"], c["depth"], seed=1 + s % 997,
                           subdivisions=c["subdivisions"], sphere_count=c["spheres"]), seed=2 + s % 991), 0, 2.6, 1.5),
}
SCALAR = ("fog", "microfacets", "demo")


def listed():
    def case(name, call, scene, width, height, spp, depth, sampler="sobol", **more):
        return dict(name=name, call=call, scene=scene, width=width, height=height, spp=spp, depth=depth,
                    sampler=sampler, **more)

    full = dict(subdivisions=8, spheres=64)   # the benchmark scene: 1,441,794 triangles
    part = dict(subdivisions=6, spheres=32)
    return [
        # an interactive viewer's frame: one sample of every pixel, read back; launches and latency
        case("frame_96x64", "frame", "cornell", 96, 64, 1, 8),
        # a driver's packet request on a ragged film with another QMC sampler, lanes to the host
        case("lanes_halton_333x251", "lanes", "cauchy", 333, 251, 3, 8, "halton"),
        # picking / visibility queries: closest hits of a list of host rays
        case("rays_200001", "rays", "mixed", 200001, 1, 1, 1, subdivisions=3, spheres=8),
        # the command line's demo render at its own defaults (scalar transport, Philox)
        case("demo_256x192_128spp", "film", "demo", 256, 192, 128, 5, "independent"),
        # a small box at a test image's size: every path in a few dozen triangles, deep paths
        case("cornell_256x256_64spp", "film", "cornell", 256, 256, 64, 8),
        # participating media: the fog-filled box, scalar transport
        case("fog_512x512_16spp", "film", "fog", 512, 512, 16, 32),
        # image reflectance: trilinear, EWA and point lookups at ray footprints
        case("textured_640x480_16spp", "film", "texture", 640, 480, 16, 8),
        # an environment image's light sampling on a ragged film
        case("sky_961x541_8spp", "film", "mixed_sky", 961, 541, 8, 16, **part),
        # a whole job from host arrays to a host film: scene upload, BVH, render, readback
        case("job_640x360_4spp", "job", "mixed", 640, 360, 4, 16, subdivisions=7, spheres=64),
        # batched views of one scene through one wavefront
        case("views_8", "views", "mixed", 512, 384, 8, 16, views=8, **part),
        # one gradient step: forward film, loss, adjoint of 512 reflectance knots
        case("gradient_512x512_32spp", "gradient", "groups", 512, 512, 32, 8),
        # the benchmark frame
        case("mixed_1080p_16spp", "film", "mixed", 1920, 1080, 16, 16, **full),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    call = rng.choice(["frame", "lanes", "rays", "film", "film", "film", "film", "job", "views", "gradient"])
    c = dict(call=call, spp=1, depth=rng.randint(4, 16), sampler=rng.choice(["sobol", "sobol", "independent", "halton"]))
    if call == "frame":
        c.update(scene=rng.choice(["cornell", "cauchy", "point"]), width=_log(rng, 48, 640), height=_log(rng, 48, 480))
    elif call == "lanes":
        c.update(scene=rng.choice(["cornell", "cauchy", "pass_through", "texture"]), width=_log(rng, 64, 480),
                 height=_log(rng, 64, 360), spp=rng.randint(1, 4))
    elif call == "rays":
        c.update(scene="mixed", width=_log(rng, 5000, 400000), height=1, depth=1, sampler="sobol",
                 subdivisions=rng.randint(2, 3), spheres=rng.randint(2, 8))
    elif call == "film":
        scene = rng.choice(["cornell", "cauchy", "texture", "pass_through", "fog", "microfacets", "demo", "mixed",
                            "mixed", "mixed_sky"])
        width, height = _log(rng, 128, 1280), _log(rng, 96, 720)
        c.update(scene=scene, width=width, height=height,
                 spp=max(1, min(64, _log(rng, 1 << 18, 1 << 23) // (width * height))))
        if scene == "demo":
            c.update(sampler="independent", depth=5)
        elif scene == "fog":
            c.update(depth=rng.randint(8, 32))
        elif scene.startswith("mixed"):
            c.update(subdivisions=rng.randint(4, 7), spheres=rng.randint(4, 64))
    elif call == "job":
        c.update(scene="mixed", width=_log(rng, 160, 960), height=_log(rng, 120, 540), spp=rng.randint(1, 4),
                 sampler="sobol", subdivisions=rng.randint(4, 7), spheres=rng.randint(4, 64))
    elif call == "views":
        c.update(scene="mixed", width=_log(rng, 256, 640), height=_log(rng, 192, 480), spp=rng.choice([4, 8]),
                 sampler="sobol", views=rng.randint(2, 8), subdivisions=rng.randint(4, 6), spheres=rng.randint(4, 32))
    else:
        c.update(scene="groups", width=_log(rng, 128, 512), height=_log(rng, 128, 512), spp=rng.choice([4, 8, 16]),
                 depth=rng.randint(4, 8), sampler="sobol")
    return c


def _settings(c, seed):
    return renderer.RenderSettings(c["width"], c["height"], samples=c["spp"], batch_size=c["spp"], seed=1 + seed % 65521,
                                   sampler=SAMPLERS[c["sampler"]])


def _build(scene):
    built = renderer.build_renderer(scene)
    if built.status != abi.RP_SUCCESS:
        raise RuntimeError(built.diagnostic)
    return built.scene


def _film(pixels):
    return torch.zeros((pixels, FILM_DOUBLES), dtype=torch.float64, device="cuda")


def _rays(c, seed):
    """Rays from above the scene to points of its ground plane, which stops those that hit
    nothing before it: origin, direction (not normalised), tmax."""
    rng = np.random.default_rng(seed)
    n = c["width"]
    o = np.stack([rng.uniform(-5, 5, n), rng.uniform(1.5, 5, n), rng.uniform(-5, 5, n)], 1)
    t = np.stack([rng.uniform(-4, 4, n), np.full(n, -1.0), rng.uniform(-4, 4, n)], 1)
    return np.concatenate([o, t - o, np.full((n, 1), np.inf)], 1).astype(np.float32)


def prepare(case, seed):
    c = case
    scene = SCENES[c["scene"]][0](c, seed)
    # a render resumes at an absolute sample, as a checkpointed or sharded one does
    state = dict(call=c["call"], settings=_settings(c, seed), seed=seed, begin=c["spp"] * (seed % 61))
    if c["call"] == "job":
        state["scene"] = scene  # host arrays; the pass builds them
        return state
    state["rs"] = rs = _build(scene)
    pixels = c["width"] * c["height"]
    if c["call"] == "frame":
        state["session"] = renderer.FrameSession(rs, renderer.FrameConfig(
            c["width"], c["height"], seed=1 + seed % 65521, sampler=SAMPLERS[c["sampler"]]))
    elif c["call"] == "lanes":
        state["request"] = renderer.RenderRequest(c["width"], c["height"], seed=1 + seed % 65521,
                                                  sample_begin=state["begin"], sample_count=c["spp"], sampler=SAMPLERS[c["sampler"]])
    elif c["call"] == "rays":
        state["rays"] = _rays(c, seed)
    elif c["call"] == "film":
        state["film"] = _film(pixels)
    elif c["call"] == "views":
        # poses from the seed; each view a little smaller than the one before it
        sizes = [(c["width"] - 23 * k, c["height"] - 13 * k) for k in range(c["views"])]
        state["views"] = [scenes.view_batch(scene, count=1, seed=seed + k, min_size=s, max_size=s, spp=(c["spp"],))[0]
                          for k, s in enumerate(sizes)]
        renderer.pack_views(state["views"])
        state["film"] = _film(sum(v.width * v.height for v in state["views"]))
        # the shape that the tuner picks for the benchmark's views
        state["request"] = renderer.BatchRequest(seed=1 + seed % 65521, wave_lanes=1 << 22, trace_block=64,
                                                 shade_block=256, blocks_per_sm=16)
    elif c["call"] == "gradient":
        state["film"] = _film(pixels)
        state["gradient"] = torch.zeros(512, dtype=torch.float32, device="cuda")
        rng = np.random.default_rng(seed)
        state["target"] = torch.from_numpy(rng.uniform(0.0, 0.5, (pixels, 3))).cuda()
    return state


def _mean(film):
    return (film[:, 0:3] + film[:, 3:6]) / (film[:, 6:7] + film[:, 7:8])


def run(state):
    s, rs = state, state.get("rs")
    if s["call"] == "frame":
        session = s["session"]
        st, frame, _, diag = session.submit(s["seed"] % 1024)
        if st != abi.RP_SUCCESS:
            raise RuntimeError(diag)
        session.wait(frame)
        _, _, xyz = session.capture(frame)
        session.release(frame)
        return xyz
    if s["call"] == "lanes":
        lanes = rs.sample(s["request"])
        if lanes.status != abi.RP_SUCCESS:
            raise RuntimeError(lanes.diagnostic)
        p = lanes.packet_samples
        return {name: p[name] for name in ("status", "pixel", "sample_low", "wavelengths", "wavelength_pdfs", "radiance")}
    if s["call"] == "rays":
        hits = rs.trace(s["rays"])
        return {"t": hits[:, 0], "b": hits[:, 1:3], "prim": np.ascontiguousarray(hits[:, 3]).view(np.int32)}
    if s["call"] == "film":
        rs.render_film_device(s["settings"], s["film"].data_ptr(), sample_begin=s["begin"], fresh=True)
        return s["film"]
    if s["call"] == "job":
        st, diag, film = renderer.render_progressive(s["scene"], s["settings"], fresh=True)
        if st != abi.RP_SUCCESS:
            raise RuntimeError(diag)
        return film.view(np.float64).reshape(-1, FILM_DOUBLES)
    if s["call"] == "views":
        # each view accumulates onto its film's committed state: a new batch starts from zero
        s["film"].zero_()
        torch.cuda.current_stream().synchronize()
        rs.render_views_device(s["views"], s["request"], s["film"].data_ptr())
        return s["film"]
    rs.render_film_device(s["settings"], s["film"].data_ptr(), fresh=True)
    d_loss = 2 * (_mean(s["film"]) - s["target"])
    torch.cuda.current_stream().synchronize()  # the renderer has a stream of its own
    rs.adjoint_device(s["settings"], list(range(16)), d_loss.data_ptr(), s["gradient"].data_ptr())
    return {"film": s["film"], "gradient": s["gradient"]}


def work(case):
    """Bytes: the scene's vertices and triangles read once, the rays read, the outputs written.
    Flops: per ray an 8-wide tree's descent to the hit (eight boxes of twelve operations a
    level) and two triangle tests of forty, per event about 600 for its two BSDF evaluations,
    light sample and four wavelengths' weights."""
    c = case
    _, triangles, rays, events = SCENES[c["scene"]]
    if "subdivisions" in c:
        triangles = 20 * 4 ** c["subdivisions"] + 2048 * c["spheres"] + 2
    pixels, samples = c["width"] * c["height"], c["width"] * c["height"] * c["spp"]
    scene_bytes = triangles * (12 + 6)  # three indices and about half a vertex a triangle
    if c["call"] == "views":
        pixels = sum((c["width"] - 23 * k) * (c["height"] - 13 * k) for k in range(c["views"]))
        samples = pixels * c["spp"]
    out = {"frame": 12 * pixels, "lanes": 80 * samples, "rays": (28 + 16) * samples}.get(c["call"], abi.FILM_PIXEL_BYTES * pixels)
    if c["call"] == "rays":
        rays, events = 1.0, 0.0
    if c["call"] == "gradient":
        rays, events = 2 * rays, 2 * events
    levels = max(1.0, math.log(triangles, 8))
    return {"bytes": scene_bytes + out, "flops": samples * (rays * (levels * 8 * 12 + 80) + events * 600)}


def exact(case, seed):
    """The rays' hit distances by a scan over every triangle in 64 bits.  The other cases are
    Monte Carlo estimates of whole paths (their 32-bit samples decide each path's turns), for
    which a 64-bit scan of every ray is out of reach in a few seconds."""
    c = case
    if c["call"] != "rays":
        return None
    scene = SCENES[c["scene"]][0](c, seed)
    device = "cuda" if torch.cuda.is_available() else "cpu"
    corners = np.concatenate([scene.positions[i.vertex_begin + scene.triangles[i.triangle_begin:i.triangle_begin + i.triangle_count].astype(np.int64)]
                              for i in scene.instances])  # identity transforms: (triangles, 3, 3)
    v = torch.from_numpy(corners.astype(np.float64)).to(device)
    e1, e2, v0 = v[:, 1] - v[:, 0], v[:, 2] - v[:, 0], v[:, 0]
    n = torch.linalg.cross(e1, e2)
    rays = torch.from_numpy(_rays(c, seed).astype(np.float64)).to(device)
    t_all = []
    chunk = max(1, (1 << 24) // v.shape[0])
    for begin in range(0, rays.shape[0], chunk):
        o, d = rays[begin:begin + chunk, None, 0:3], rays[begin:begin + chunk, None, 3:6]
        s = v0[None] - o
        det = (d * n[None]).sum(-1)
        t = (s * n[None]).sum(-1) / det
        q = torch.linalg.cross(s, d.expand_as(s))
        u = (q * e2[None]).sum(-1) / det
        w = -(q * e1[None]).sum(-1) / det
        inside = (u >= 0) & (w >= 0) & (u + w <= 1) & (t > 0)
        t_all.append(torch.where(inside, t, torch.inf).amin(1))
    return {"t": torch.cat(t_all).cpu().numpy(), "b": None, "prim": None}
