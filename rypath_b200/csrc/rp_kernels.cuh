// Wavefront kernels of the hero path tracer and the device film reduction.
#pragma once

#include "rp_transport.cuh"
#include "rp_walk.cuh"

namespace rp {

constexpr int kTraceBlock = 128;

// Warp-aggregated append to a device queue: one atomicAdd per warp.  Every lane of the warp
// must call this together (the shade kernel runs a warp-uniform trip count).
RP_DEV u32 warp_append(u32 *counter, bool want) {
    const u32 ballot = __ballot_sync(0xffffffffu, want);
    const int lane = threadIdx.x & 31;
    u32 base = 0;
    if (lane == 0 && ballot)
        base = atomicAdd(counter, __popc(ballot));
    base = __shfl_sync(0xffffffffu, base, 0);
    return base + __popc(ballot & ((1u << lane) - 1));
}

// rypath_render_packets prologue (shaders/render.metal:2424-2460) + packet_pt_initialize
// (shaders/packet_pt_step.h:84-115) for request lane `lane`, stored in pool slot `slot`.
RP_DEV void raygen_lane(const DeviceScene &s, const RasterCam &cam, const WaveParams &p, u32 lane, u32 slot,
                        PathPool &pool) {
    {
        const BeginSample b = begin_sample(s, p, lane);
        V4 lambda, pdf;
        sample_wavelengths(sample_uniform(p, b.words.z), s.hero_mode, lambda, pdf);
        V3 o, d;
        primary_ray_from(s, cam, p, b, o, d);
        u32 flags = 15u | F_ROULETTE;
        if (!finite3(o) || !finite3(d))
            flags = set_status(flags, 2) | F_COMPLETE;
        pool.ident(slot) = make_uint4(b.pixel, b.sample_low, b.sample_high, flags);
        pool.index(slot) = make_uint4(u32(b.index), u32(b.index >> 32), 0, 0);
        pool.lambda(slot) = to_float4(lambda);
        pool.lambda_pdf(slot) = to_float4(pdf);
        pool.radiance(slot) = make_float4(0, 0, 0, 0);
        pool.ray_o(0, slot) = make_float4(o.x, o.y, o.z, 0);
        pool.ray_d(0, slot) = make_float4(d.x, d.y, d.z, 0);
        pool.vertex(0, slot)[0] = make_float4(o.x, o.y, o.z, 0);
        pool.queue[0][slot] = slot;
        if (pool.lane_closest) {
            pool.lane_closest[slot] = 0;
            pool.lane_shadow[slot] = 0;
        }
        if (pool.hist) {
            pool.hist[slot] = empty_history();
            pool.adj_w[slot] = adjoint_lane_weight(pool, b.pixel, lambda, pdf);
        }
    }
}
// Issue-bound by the draw words.  The first event uses constants for the initial throughput, eta
// scale and density, which are not written: mixed scene 1080p, 16 spp 81.8 -> 80.3 ms, with the
// camera's draw block from a table.
__global__ void k_raygen(const __grid_constant__ DeviceScene s, const __grid_constant__ WaveParams p, PathPool pool) {
    const RasterCam cam{s.origin, s.forward, s.right, s.up};
    if (blockIdx.x == 0 && threadIdx.x == 0)
        pool.counters[0] = p.lanes;
    for (u32 lane = blockIdx.x * blockDim.x + threadIdx.x; lane < p.lanes; lane += gridDim.x * blockDim.x)
        raygen_lane(s, cam, p, lane, lane, pool);
}

// Hit records the shade kernels read as a failed event (rp_sample_status 3, 4, 2).
constexpr u32 kHitInvalid = 0xfffffffeu, kHitExhausted = 0xfffffffdu, kHitArithmetic = 0xfffffffcu;

// A hit on a pass-through or mix-root instance, resolved before shading
// (shaders/packet_pt_event_body.inc:100-205): the same validity checks and surface point as
// the event, then either a crossing (at most boundary_limit in a row, each a new walk from
// the spawned origin, which is written to ray_o) or the mix resolution (the resolved material
// written to pool.material).  Returns the family to bin (3 for a failure or a miss) and sets
// `prim` to the primitive or failure code to record.
template <bool Count, int Stack>
__device__ __noinline__ u32 resolve_hit(const DeviceScene &s, const PathPool &pool, int in, u32 path, V3 ro, V3 rd, Hit &h,
                                        u32 &prim, uint2 *stack, int stride, u32 boundary_limit, u32 &nodes, u32 &tris,
                                        u32 &rays) {
    u32 crossings = 0;
    bool moved = false;
    u32 family = 3;
    for (;;) {
        if (!isfinite(h.t) || h.t < 0 || !isfinite(h.b1) || !isfinite(h.b2)) {
            prim = kHitInvalid;
            break;
        }
        const u32 inst = s.tri_instance[h.prim];
        const DInstance &in = s.instances[inst];
        if (in.material >= s.material_count) {
            prim = kHitInvalid;
            break;
        }
        SurfacePoint pt;
        if (!hit_surface_point(s, h.prim, inst, s.tri_local[h.prim], h.b1, h.b2, pt)) {
            prim = kHitArithmetic;
            break;
        }
        if (in.resolve & kPassThrough) {
            V3 origin;
            if (crossings++ >= boundary_limit) {
                prim = kHitExhausted;
                break;
            }
            if (!spawn_boundary(ro, rd, h.t, pt, rd, origin)) {
                prim = kHitArithmetic;
                break;
            }
            ro = origin;
            moved = true;
            ++rays;
            if (!walk_closest<Count, Stack, true>(s, ro, rd, __int_as_float(0x7f800000), h, stack, stride, nodes, tris)) {
                prim = kHitInvalid;
                break;
            }
            prim = h.prim;
            if (prim == kNone)
                break;
            family = __ldg(s.tri_family + prim);
            if (family != kResolveFamily)
                break;
            continue;
        }
        u32 material = in.material;
        const u32 status = resolve_mix(s, pt.position, -rd, material);
        if (status != 0) {
            prim = status == 2 ? kHitArithmetic : kHitInvalid;
            break;
        }
        pool.material[path] = material;
        prim = h.prim;
        family = s.materials[material].scattering;
        break;
    }
    if (moved)
        pool.ray_o(in, path) = make_float4(ro.x, ro.y, ro.z, 0);
    return prim >= kHitArithmetic || prim == kNone ? 3u : family;
}

// Closest-hit queries for the active queue; each path is then appended to the bin of the
// BSDF family it hit (0 diffuse, 1 conductor, 2 dielectric, 3 miss or failed query), so the
// shade stage runs one specialised kernel per family ("material-sorted shading").
struct TraceRays {
    const DeviceScene &s;
    const PathPool &pool;
    const u32 *queue;
    int in;
    u32 *event;
    StagedAppend bins;
    u32 path;

    template <class W> RP_DEV bool load(u32 i, W &w) {
        path = queue[i];
        if (pool.ident(path).w & F_COMPLETE)
            return false;
        const float4 o = pool.ray_o(in, path), d = pool.ray_d(in, path);
        w.start(s, v3(o.x, o.y, o.z), v3(d.x, d.y, d.z), __int_as_float(0x7f800000));
        return true;
    }
    template <class W> RP_DEV void finish(bool done, const W &w) {
        u32 family = 4;
        if (done) {
            const u32 prim = w.ok ? w.h.prim : kHitInvalid;
            family = (!w.ok || w.h.prim == kNone) ? 3u : u32(__ldg(s.tri_family + w.h.prim));
            pool.hit(path) = make_float4(w.h.t, w.h.b1, w.h.b2, __uint_as_float(prim));
        }
#pragma unroll
        for (u32 f = 0; f < 4; ++f)
            bins.push(f, family == f, path, event + kBinCount + f, pool.bins + size_t(f) * pool.bin_capacity);
    }
    RP_DEV void flush() {
#pragma unroll
        for (u32 f = 0; f < 4; ++f)
            bins.flush(f, event + kBinCount + f, pool.bins + size_t(f) * pool.bin_capacity);
    }
};
// Blocks per SM of the walk kernels: with the short stack, eight of 128 threads (64 registers)
// for the plain form and six (80) for the streaming one, whose state spills at 64.
constexpr int walk_blocks(int block, int stack, bool stream) {
    return stack > kShortStack ? 1 : (stream ? 768 : 1024) / block;
}
// Stack: traversal stack entries per thread (kShortStack for shallow trees, whose walks then
// fit eight 128-thread blocks per SM).
// Resolve: the scene has pass-through, mix-root or procedural instances (resolve_hit).
// Stream: walk_stream, else a ray a thread at a time (use_stream says when).
template <bool Count, int Block = kTraceBlock, int Stack = kStackDepth, bool Resolve = false, bool Stream = false>
__global__ void __launch_bounds__(Block, walk_blocks(Block, Stack, Stream))
    k_trace(const __grid_constant__ DeviceScene s, PathPool pool, int in, u32 boundary_limit) {
    __shared__ uint2 stack[Stack * Block];
    const u32 count = pool.counters[in];
    u32 *event = pool.event(in);
    if (blockIdx.x == 0 && threadIdx.x == 0)
        pool.counters[in ^ 1] = 0;
    if constexpr (Stream) {
        static_assert(!Count && !Resolve);
        __shared__ u32 stage[Block / 32 * 4 * kStageEntries];
        TraceRays io{s, pool, pool.queue[in], in, event, {stage + (threadIdx.x >> 5) * 4 * kStageEntries, 0}, 0};
        walk_stream<Walker<false, Stack>>(s, count, event + kTraceNext, stack + threadIdx.x, Block, io);
        return;
    }
    const u32 *queue = pool.queue[in];
    u32 nodes = 0, tris = 0, rays = 0;
    const u32 stride = gridDim.x * blockDim.x;
    const u32 trips = (count + stride - 1) / stride;
    const int lane = threadIdx.x & 31;
    for (u32 trip = 0; trip < trips; ++trip) {
        const u32 i = trip * stride + blockIdx.x * blockDim.x + threadIdx.x;
        u32 family = 4, path = 0;
        if (i < count) {
            path = queue[i];
            if (!(pool.ident(path).w & F_COMPLETE)) {
                const float4 o = pool.ray_o(in, path), d = pool.ray_d(in, path);
                const u32 walks_before = rays;
                Hit h;
                const bool ok = walk_closest<Count, Stack, Resolve>(s, v3(o.x, o.y, o.z), v3(d.x, d.y, d.z),
                                                                    __int_as_float(0x7f800000), h, stack + threadIdx.x,
                                                                    Block, nodes, tris);
                ++rays;
                u32 prim = ok ? h.prim : kHitInvalid;
                family = (!ok || h.prim == kNone) ? 3u : u32(__ldg(s.tri_family + h.prim));
                if (Resolve && family == kResolveFamily)
                    family = resolve_hit<Count, Stack>(s, pool, in, path, v3(o.x, o.y, o.z), v3(d.x, d.y, d.z), h, prim,
                                                       stack + threadIdx.x, Block, boundary_limit, nodes, tris, rays);
                pool.hit(path) = make_float4(h.t, h.b1, h.b2, __uint_as_float(prim));
                if (Count && pool.lane_closest)
                    pool.lane_closest[path] += rays - walks_before;
            }
        }
        const u32 peers = __match_any_sync(0xffffffffu, family);
        const int leader = __ffs(peers) - 1;
        u32 base = 0;
        if (lane == leader && family < 4)
            base = atomicAdd(event + kBinCount + family, __popc(peers));
        base = __shfl_sync(0xffffffffu, base, leader);
        if (family < 4)
            pool.bins[size_t(family) * pool.bin_capacity + base + __popc(peers & ((1u << lane) - 1))] = path;
    }
    if (Count) {
        atomicAdd(pool.stats + 0, (unsigned long long)nodes);
        atomicAdd(pool.stats + 1, (unsigned long long)tris);
        atomicAdd(pool.stats + 2, (unsigned long long)rays);
    }
}

// The warps of a block meet between two phases of a long straight run of code, so that a line of
// instructions fetched for one serves them all: the shade kernels run some four thousand
// instructions an event once each, and their warps, left to drift apart, spent up to 6.9 of 17
// cycles an instruction waiting for instructions (0.9 so; of a pass, the two kernels' part 24.8 -> 13.4
// ms in the textured box, 14.0 -> 12.1 in the Cornell box).  Blocks of 256 serve better than of 128 or 512.
template <bool Sync> RP_DEV void phase() {
    if (Sync)
        __syncthreads();
}
// One hero event of path `path` after its closest hit (shaders/packet_pt_event_body.inc:11-461),
// a hit of BSDF family F (3: no surface -- environment or a failed query).  keep: the path
// goes on; nee: its event left a light-sample request.  in: the parity of its queue;
// event_index: events before this one (every path of the wave has had as many).  Sync: the whole block calls this
// (`active` clear where it has no path), and its warps meet between the phases of the event.
template <int F, bool Adjoint, bool Img, bool Sync>
RP_DEV void shade_path(const DeviceScene &s, const WaveParams &p, const PathPool &pool, int in, u32 event_index,
                       bool active, u32 path, float *sgrad, bool &keep, bool &nee) {
    const u32 capacity = s.max_depth + 2;
    uint4 ident = make_uint4(0, 0, 0, 0);
    if (active)
        ident = pool.ident(path);
    u32 flags = ident.w;
    active = active && !(flags & F_COMPLETE);
    {
        u32 cnt = event_index + 1; // vertices so far, the camera's included
        // at the first event the throughput, eta scale and density are the initial ones
        V4 lambda = v4(0), beta = v4(1), eta_scale = v4(1);
        Density density = initial_density();
        u64 index = 0;
        V3 ro = v3(0, 0, 0), rd = v3(0, 0, 0);
        float4 hit = make_float4(0, 0, 0, 0);
        if (active) { // a thread without a path has no record to read: another's is written meanwhile
            const uint4 index2 = pool.index(path);
            index = (u64(index2.y) << 32) | index2.x;
            lambda = from_float4(pool.lambda(path));
            if (event_index) {
                beta = from_float4(pool.beta(path));
                eta_scale = from_float4(pool.eta_scale(path));
                density = event_density(pool, in, path, event_index);
            }
            const float4 ro4 = pool.ray_o(in, path), rd4 = pool.ray_d(in, path);
            ro = v3(ro4.x, ro4.y, ro4.z);
            rd = v3(rd4.x, rd4.y, rd4.z);
            hit = pool.hit(path);
        }
        bool roulette = (flags & F_ROULETTE) != 0;
        u32 active_mask = flags & F_MASK;
        u32 status = get_status(flags);
        const Density direct_density = density;
        V4 direct_beta = beta;
        bool direct_allowed = true;
        const u32 old_count = cnt;
        bool terminated = true;
        // current vertex
        u32 ctype = kSurface, cinst = kNone, clocal = 0, clight = kNone, cmat = kNone;
        SurfacePoint cp;
        cp.position = cp.error = cp.geometric_normal = cp.shading_normal = v3(0, 0, 0);
        cp.inverse_area_pdf = 0;
        Frame cframe;
        HeroBsdf cbsdf;
        cbsdf.kind = 0;
        cbsdf.active_mask = active_mask;
        cbsdf.g = {0, 0, true};
        V4 cbeta = beta;
        V3 cwo = v3(0, 0, 0), swo = v3(0, 0, 0);
        bool cdelta = false, connectible = false;
        bool go = false; // the event goes on to its next phase
        if (active) do {
            if (cnt >= capacity || !nonzero4(beta))
                break;
            if (!finite3(ro) || !finite3(rd) || !finite_nonnegative4(beta)) {
                status = 2;
                break;
            }
            const u32 prim = __float_as_uint(hit.w);
            if (prim >= kHitArithmetic && prim != kNone) {
                status = prim == kHitInvalid ? 3u : prim == kHitExhausted ? 4u : 2u;
                break;
            }
            if (prim == kNone) {
                ctype = kEnvironment;
                clight = s.environment_light;
                cp.position = ro + rd;
                cp.geometric_normal = -rd;
                cp.shading_normal = -rd;
                cwo = -rd;
                cbeta = beta;
                connectible = true;
                ++cnt;
                break;
            }
            if constexpr (F == 3) {
                status = 3; // a surface hit never reaches the no-surface bin
                break;
            } else {
                const float t = hit.x, b1 = hit.y, b2 = hit.z;
                if (!isfinite(t) || t < 0 || !isfinite(b1) || !isfinite(b2) || prim >= s.prim_count) {
                    status = 3;
                    break;
                }
                cinst = s.tri_instance[prim];
                clocal = s.tri_local[prim];
                const DInstance &instance = s.instances[cinst];
                if (instance.material >= s.material_count) {
                    status = 3;
                    break;
                }
                // a mix root's hit was resolved by the closest-hit kernel
                cmat = (instance.resolve & kMixRoot) ? pool.material[path] : instance.material;
                ctype = kSurface;
                clight = instance.emission == kNone ? kNone : instance.emitter_begin + clocal;
                cwo = -rd;
                if (!hit_surface_point(s, prim, cinst, clocal, b1, b2, cp)) {
                    status = 2;
                    break;
                }
                const DMaterial material = s.materials[cmat];
                // an image reflectance reads its texture at the hit's footprint
                // (shaders/packet_pt_event_body.inc:147-163, packet_walk.h:39-49)
                RgbPolynomial image_rgb;
                bool image = false;
                if constexpr (F == 0) {
                    if (Img && s.img.textured && material.kind == 3 && material.image_texture < s.img.texture_count) {
                        F2 st, dstdx, dstdy;
                        if (!texture_context(s, p, ident.x, ident.y, ident.z, cinst, clocal, b1, b2,
                                             cp.geometric_normal, rd, cnt - 1, st, dstdx, dstdy)) {
                            status = 2;
                            break;
                        }
                        image_rgb = rgb_polynomial(
                            s.img.rgb_table, image_reflectance_rgb(s.img, material.image_texture, st, dstdx, dstdy));
                        image = true;
                    }
                }
                if (!shading_frame(cp.shading_normal, cframe) ||
                    !prepare_bsdf<F>(s, material, lambda, active_mask, cbsdf, image ? &image_rgb : nullptr)) {
                    status = 2;
                    break;
                }
                V3 ray_position, ray_error;
                ray_point(ro, rd, t, cp.curved, ray_position, ray_error);
                cp.error = cp.error + (vabs(cp.position - ray_position) + ray_error);
                if (!finite3(cp.error)) {
                    status = 2;
                    break;
                }
                cbeta = beta;
                connectible = hero_connectible(cbsdf);
                ++cnt;
                if (cnt == capacity)
                    break;
                if (cnt - 2 >= p.emergency_limit) {
                    status = 1;
                    break;
                }
                go = true;
            }
        } while (false);
        if constexpr (F != 3) {
            phase<Sync>();
            uint4 draws;
            if (go) {
                // only a dielectric reads the lobe word, a smooth one only that of the
                // three, and the first event no roulette word
                const bool survival = roulette && cnt > 2;
                const u32 set = F == 2 ? (cbsdf.g.smooth ? (survival ? kDrawXW : kDrawX) : kDrawAll)
                                       : (survival ? kDrawYZW : kDrawYZ);
                draws = draw_words(s, p, ident.x, ident.y, ident.z, index, 4 + cnt - 2, set);
                swo = to_local(cframe, cwo);
                cbsdf.active_mask = active_mask;
                direct_allowed = hero_continue(beta, eta_scale, roulette, cnt - 1, sample_uniform(p, draws.w));
                direct_beta = beta;
                connectible = hero_connectible(cbsdf);
                go = direct_allowed;
            }
            phase<Sync>();
            if (go) do {
                const HeroSample proposed = hero_sample_k<F>(cbsdf, swo, sample_uniform(p, draws.x),
                                                        sample_uniform(p, draws.y), sample_uniform(p, draws.z));
                bool cont_valid = proposed.valid;
                if (proposed.valid && proposed.accepted) {
                    const Update adv = advance(direct_density, beta, proposed.numerator, proposed.pdf);
                    cont_valid = adv.valid;
                    if (adv.valid) {
                        beta = adv.beta;
                        density = adv.density;
                    }
                    hero_account_eta(eta_scale, roulette, proposed.eta, proposed.transmission);
                    active_mask = 1;
    #pragma unroll
                    for (int k = 1; k < 4; ++k)
                        if (density.lane[k].fraction > 0 || (fbits(beta.v[k]) & 0x7fffffffu))
                            active_mask |= 1u << k;
                }
                if (!cont_valid) {
                    status = 2;
                    break;
                }
                if (!proposed.accepted)
                    break;
                V3 wi = to_world(cframe, proposed.wi);
                if (!unit_vector(wi, wi)) {
                    status = 2;
                    break;
                }
                if (!finite_nonnegative4(beta)) {
                    status = 2;
                    break;
                }
                if (proposed.delta)
                    cdelta = true;
                const V3 origin = offset_point(cp.position, cp.error, cp.geometric_normal, wi);
                if (!finite3(origin)) {
                    status = 2;
                    break;
                }
                ro = origin;
                rd = wi;
                terminated = false;
            } while (false);
        }
        phase<Sync>();
        bool complete = terminated || status != 0 || cnt >= capacity || !nonzero4(beta);
        // latest vertex (the previous event's) for MIS; what only a weighted emission reads of
        // it is loaded there
        Latest latest;
        latest.kind = (flags >> F_LKIND_SHIFT) & 3u;
        latest.mask = (flags >> F_LMASK_SHIFT) & 15u;
        latest.delta = (flags & F_LDELTA) != 0;
        latest.smooth = (flags & F_LSMOOTH) != 0;
        if (cnt != old_count && status == 0) {
            // hero_endpoint (shaders/hero_pt_helpers.h:157-184)
            V4 rad = v4(0);
            bool emission_ok = true;
            if (ctype == kEnvironment) {
                if (Img && s.img.env_image != kNone) {
                    rad = environment_image_radiance4(s.img, rd, lambda);
                } else if (s.environment != kNone) {
#pragma unroll
                    for (int k = 0; k < 4; ++k)
                        rad.v[k] = spectrum(s, s.environment, lambda.v[k]);
                }
                emission_ok = finite_nonnegative4(rad);
            } else {
                const DInstance &instance = s.instances[cinst];
                V3 delta = v3(0, 0, 0);
                if (instance.emission != kNone) {
                    const float4 lp4 = pool.vertex(in, path)[0];
                    delta = v3(lp4.x, lp4.y, lp4.z) - cp.position;
                }
                if (!zero3(delta)) {
                    const V3 dir = normalize3(delta);
                    if (s.emission_two_sided[instance.emission] || dot(cp.geometric_normal, dir) > 0) {
                        const u32 off = instance.emission * 471u;
#pragma unroll
                        for (int k = 0; k < 4; ++k)
                            rad.v[k] = cp.inverse_area_pdf == 0 ? 0.f : spectrum(s, off, lambda.v[k]);
                        emission_ok = finite_nonnegative4(rad);
                    }
                }
            }
            V4 endpoint = v4(0);
            if (!emission_ok) {
                status = 2;
            } else {
                const V4 value = mul4(cbeta, rad);
                if (cnt <= 2 || latest.delta || !nonzero4(value)) {
                    endpoint = value;
                } else {
                    const float4 *vertex = pool.vertex(in, path);
                    const float4 lp4 = vertex[0], ln4 = vertex[1];
                    latest.position = v3(lp4.x, lp4.y, lp4.z);
                    latest.shading_normal = v3(ln4.x, ln4.y, ln4.z);
                    latest.alpha_x = lp4.w;
                    latest.alpha_y = ln4.w;
                    latest.param = from_float4(vertex[2]);
                    latest.k = latest.kind == 1 ? from_float4(vertex[3]) : v4(0);
                    const float4 pre = pool.vertex(in ^ 1, path)[0]; // the vertex before it
                    const Density previous_density = event_density(pool, in ^ 1, path, event_index - 1);
                    bool ok;
                    const V4 bsdf_pdf = represented_pdf<-1>(latest_bsdf(latest), latest.shading_normal, latest.position,
                                                        v3(pre.x, pre.y, pre.z), ctype == kEnvironment,
                                                        ctype == kEnvironment ? rd : cp.position, ok);
                    // hero_history_light_pdf / direct_pdf (shaders/packet_transport.h:740-758)
                    float lpdf = 0;
                    const float selection = light_pmf(s, latest.position, latest.shading_normal, clight);
                    if (ctype == kEnvironment) {
                        // the constant environment has no unidirectional proposal;
                        // the image's is its compensated table
                        lpdf = (Img && s.img.env_image != kNone) ? environment_image_pdf(s.img, rd, true) * selection
                                                        : 0.0f * selection;
                    } else {
                        const V3 dl = cp.position - latest.position;
                        if (dot(dl, dl) > 0 && nonzero3(cp.geometric_normal) && clight < s.emitter_count)
                            lpdf = selection * light_geometry_pdf(s, clight, latest.position,
                                                                  latest.shading_normal, cp);
                    }
                    if (!ok || !hero_weight(previous_density, value, ok ? bsdf_pdf : v4(__int_as_float(0x7fffffff)),
                                            v4(lpdf), endpoint))
                        status = 2;
                }
            }
            // radiance is finite and nonnegative while its path lives; a zero endpoint leaves it
            bool radiance_ok = true;
            if (endpoint.v[0] != 0 || endpoint.v[1] != 0 || endpoint.v[2] != 0 || endpoint.v[3] != 0) {
                const V4 radiance = add4(from_float4(pool.radiance(path)), endpoint);
                pool.radiance(path) = to_float4(radiance);
                radiance_ok = finite_nonnegative4(radiance);
            }
            if (Adjoint) {
                // replay: the emission's gradient over the vertices before this one,
                // then this diffuse vertex joins the history of what follows it
                uint4 h = pool.hist[path];
                if (status == 0 && nonzero4(endpoint))
                    adjoint_accumulate(s, pool, sgrad, h, lambda, endpoint, pool.adj_w[path]);
                if (F == 0 && ctype == kSurface && status == 0) {
                    const u32 m = cmat;
                    if (__ldg(pool.adj_slot + m) != kNone) {
                        h = history_push(h, m);
                        pool.hist[path] = h;
                    }
                }
            }
            // hero_direct (shaders/hero_pt_helpers.h:185-221) runs in the light-sample kernel
            // (k_nee), from the request this event leaves; its failures fail the path there.
            nee = F != 3 && status == 0 && cnt < capacity && direct_allowed && ctype == kSurface && connectible;
            if (!radiance_ok)
                status = 2;
            if (status != 0) {
                complete = true;
                nee = false;
            }
            if (nee) {
                float4 *request = pool.request(path);
                request[0] = make_float4(cp.geometric_normal.x, cp.geometric_normal.y, cp.geometric_normal.z, 0);
                request[1] = make_float4(cp.error.x, cp.error.y, cp.error.z, 0);
                request[2] = to_float4(direct_beta);
            }
        }
        phase<Sync>();
        if (!active)
            return;
        // A complete path is read again only for its identity, status and radiance (the shadow
        // walk, the film and the packet results) and, with a light sample, its vertex, so the
        // rest of its state is not written back.
        if (cnt != old_count) {
            // preceding = latest; latest = current (shaders/packet_pt_event_body.inc:453-460)
            if (!complete || nee) {
                float4 *vertex = pool.vertex(in ^ 1, path);
                vertex[0] = make_float4(cp.position.x, cp.position.y, cp.position.z, cbsdf.g.alpha_x);
                vertex[1] = make_float4(cp.shading_normal.x, cp.shading_normal.y, cp.shading_normal.z, cbsdf.g.alpha_y);
                vertex[2] = make_float4(cbsdf.param[0], cbsdf.param[1], cbsdf.param[2], cbsdf.param[3]);
                if (F == 1)
                    vertex[3] = make_float4(cbsdf.k[0], cbsdf.k[1], cbsdf.k[2], cbsdf.k[3]);
            }
            flags &= ~(F_LDELTA | (3u << F_LKIND_SHIFT) | (15u << F_LMASK_SHIFT) | F_LSMOOTH);
            flags |= (cdelta ? F_LDELTA : 0u) | ((cbsdf.kind & 3u) << F_LKIND_SHIFT) |
                     ((cbsdf.active_mask & 15u) << F_LMASK_SHIFT) | (cbsdf.g.smooth ? F_LSMOOTH : 0u);
        }
        flags = (flags & ~(F_MASK | F_ROULETTE)) | active_mask | (roulette ? F_ROULETTE : 0u);
        flags = set_status(flags, status) | (complete ? F_COMPLETE : 0u);
        ident.w = flags;
        pool.ident(path) = ident;
        if (!complete) {
            pool.beta(path) = to_float4(beta);
            float4 f;
            int4 e;
            store_density(density, f, e);
            pool.dens_f(in ^ 1, path) = f;
            pool.dens_e(in ^ 1, path) = e;
            if (F == 2 || event_index == 0)
                pool.eta_scale(path) = to_float4(eta_scale); // only transmission changes it
            pool.ray_o(in ^ 1, path) = make_float4(ro.x, ro.y, ro.z, 0);
            pool.ray_d(in ^ 1, path) = make_float4(rd.x, rd.y, rd.z, 0);
        }
        keep = !complete;
    }
}
// shade_path of the paths in the bin of family F.
// Adjoint: the path-replay adjoint hooks are compiled in (the plain forward kernel carries none
// of their registers).  512 resident threads per SM cap the registers at 128, which the plain
// forms keep to without spilling (200 to 300 bytes a thread before the event's state was cut:
// mixed scene 1080p, 16 spp 91.9 against 84.5 ms).
// Img: the scene has image reflectance or an environment image (their code is compiled out of
// the plain kernels).
template <int F, int Block = 128, bool Adjoint = false, bool Img = true>
__global__ void __launch_bounds__(Block, 512 / Block) k_shade(const __grid_constant__ DeviceScene s,
                                                              const __grid_constant__ WaveParams p, PathPool pool, int in,
                                                              u32 event_index) {
    extern __shared__ float sgrad[]; // adjoint only
    if (Adjoint)
        adjoint_begin(pool, sgrad);
    u32 *event = pool.event(in);
    if (F == 3 && blockIdx.x == 0 && threadIdx.x < kEventCounters)
        pool.event(in ^ 1)[threadIdx.x] = 0;
    const u32 count = event[kBinCount + F];
    const u32 *queue = pool.bins + size_t(F) * pool.bin_capacity;
    u32 *out_queue = pool.queue[in ^ 1];
    u32 *out_count = pool.counters + (in ^ 1);
    // uniform trip count so warp-level appends see every lane of the warp
    const u32 stride = gridDim.x * blockDim.x;
    const u32 trips = (count + stride - 1) / stride;
    for (u32 trip = 0; trip < trips; ++trip) {
        const u32 i = trip * stride + blockIdx.x * blockDim.x + threadIdx.x;
        bool keep = false, nee = false;
        u32 path = 0;
        const bool active = i < count;
        if (active)
            path = queue[i];
        shade_path<F, Adjoint, Img, true>(s, p, pool, in, event_index, active, path, sgrad, keep, nee);
        const u32 slot = warp_append(out_count, keep);
        if (keep)
            out_queue[slot] = path;
        if (F != 3) {
            const u32 nslot = warp_append(event + kNeeCount + F, nee);
            if (nee)
                pool.nee_queue[size_t(F) * pool.bin_capacity + nslot] = path;
        }
    }
    if (Adjoint)
        adjoint_end(pool, sgrad);
}

// The light sample of one hero event (hero_direct, shaders/hero_pt_helpers.h:185-221) of a
// path whose event (of BSDF family F) asked for one: light selection, the light's point and
// radiance, the BSDF on the light direction, the balance weight, and the visibility segment
// (shadow set).  Its own failures (invalid arithmetic) fail the path.  Split
// from the shade kernel, which leaves the request, so that each kernel
// holds half the live state.
template <int F, bool Img, bool Sync>
RP_DEV void nee_path(const DeviceScene &s, const WaveParams &p, const PathPool &pool, int in, u32 event_index, bool active,
                     u32 path, bool &shadow, float4 &sh_o, float4 &sh_d, float4 &sh_c, float4 &sh_t) {
    uint4 ident;
    u64 index;
    V4 lambda;
    SurfacePoint cp;
    HeroBsdf cbsdf;
    V3 cwo, previous;
    V4 direct_beta;
    Density direct_density;
    if (active) { // a thread without a path has no record to read: another's is written meanwhile
        ident = pool.ident(path);
        const uint4 index2 = pool.index(path);
        index = (u64(index2.y) << 32) | index2.x;
        lambda = from_float4(pool.lambda(path));
        read_nee_request<F>(pool, in, event_index, path, ident.w, cp, cbsdf, cwo, previous, direct_beta, direct_density);
    }
    u32 status = 0;
    // the light-sample draw: its first word selects the light; the next two, a point on an
    // area light, are drawn only when an area light was selected (the same words either way)
    const u32 block = 133 + event_index;
    // sample_li (shaders/packet_transport.h:470-553)
    float selected_pmf = 0; // light_pmf of the selected light
    Selected choice{kNone, 0};
    bool env_image = false;
    if (active) {
        const float u0 = sample_uniform(p, draw_words(s, p, ident.x, ident.y, ident.z, index, block, kDrawX).x);
        choice = light_sample<true>(s, cp.position, cp.shading_normal, u0, selected_pmf);
        env_image = Img && s.img.env_image != kNone && choice.light == s.environment_light;
    }
    phase<Sync>();
    V4 lbeta = v4(0);
    float spdf = 0, geometry_pdf = 0; // geometry_pdf: light_geometry_pdf of the sampled point
    bool li_ok = true, delta_light = false;
    SurfacePoint lp;
    lp.position = lp.error = lp.geometric_normal = lp.shading_normal = v3(0, 0, 0);
    lp.inverse_area_pdf = 0;
    V3 direction = v3(0, 0, 1);
    const u32 sel = choice.light;
    if (active && choice.pmf > 0) {
        float u1 = 0, u2 = 0;
        if (choice.light < s.emitter_count || env_image) {
            const uint4 w = draw_words(s, p, ident.x, ident.y, ident.z, index, block, kDrawYZ);
            u1 = sample_uniform(p, w.y);
            u2 = sample_uniform(p, w.z);
        }
        V4 lrad = v4(0);
        if (sel < s.emitter_count) {
            if (!light_geometry_sample(s, sel, cp.position, cp.shading_normal, u1, u2, lp, spdf)) {
                li_ok = false;
            } else {
                geometry_pdf = spdf;
                spdf *= choice.pmf;
                const V3 dl = lp.position - cp.position;
                const float d2 = dot(dl, dl);
                if (lp.inverse_area_pdf == 0 || !(d2 > 0)) {
                    spdf = 0;
                } else {
                    direction = dl * (1.0f / sqrtf(d2));
                    const DInstance &li = s.instances[s.emitter_instance[sel]];
                    if (s.emission_two_sided[li.emission] || dot(lp.geometric_normal, -direction) > 0) {
#pragma unroll
                        for (int k = 0; k < 4; ++k)
                            lrad.v[k] = spectrum(s, li.emission * 471u, lambda.v[k]);
                    }
                    li_ok = finite_nonnegative4(lrad);
                }
            }
        } else if (sel < s.emitter_count + s.positional_count) {
            const DPositional &L = s.positional[sel - s.emitter_count];
            delta_light = true;
            lp.position = v3(L.position[0], L.position[1], L.position[2]);
            const V3 dl = lp.position - cp.position;
            const float d2 = dot(dl, dl);
            if (!(d2 > 0)) {
                spdf = 0;
            } else {
                direction = dl * (1.0f / sqrtf(d2));
                float falloff = 1;
                const bool lit = positional_falloff(L, direction, falloff);
                li_ok = lit;
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    float intensity = spectrum(s, L.spectrum, lambda.v[k]);
                    if (lit && !apply_falloff(L, falloff, intensity))
                        li_ok = false;
                    lrad.v[k] = intensity / d2;
                }
                spdf = choice.pmf;
            }
        } else if (env_image) {
            // the environment image's compensated table (shaders/packet_transport.h:536-552)
            float epdf = 0;
            if (!sample_environment_image(s.img, u1, u2, true, direction, epdf)) {
                li_ok = false;
            } else {
                lrad = environment_image_radiance4(s.img, direction, lambda);
                spdf = epdf * choice.pmf;
                lp.position = cp.position + (2 * s.scene_radius) * direction;
                lp.geometric_normal = lp.shading_normal = -direction;
            }
        } else {
            spdf = 0; // constant environment: pdf 0 for unidirectional PT
        }
        if (li_ok)
            lbeta = spdf > 0 ? V4{{lrad.v[0] / spdf, lrad.v[1] / spdf, lrad.v[2] / spdf, lrad.v[3] / spdf}} : v4(0);
        li_ok = li_ok && finite_nonnegative4(lbeta);
    }
    if (active && (!li_ok || !isfinite(spdf) || spdf < 0))
        status = 2;
    bool go = active && status == 0 && spdf > 0 && nonzero4(lbeta);
    phase<Sync>();
    Frame cframe;
    V4 value = v4(0);
    if (go) {
        shading_frame(cp.shading_normal, cframe); // succeeded in the shade kernel
        const HeroEval e = hero_evaluate_k<F == 3 ? 0 : F>(cbsdf, to_local(cframe, cwo), to_local(cframe, direction));
        if (!e.valid)
            status = 2;
        else
            value = scale4(mul4(mul4(direct_beta, e.f), lbeta), fabsf(dot(cp.shading_normal, direction)));
        go = e.valid && nonzero4(value);
    }
    phase<Sync>();
    if (go) {
        V4 contribution = value;
        bool weight_ok = true;
        if (!delta_light) {
            const float sel_pmf = selected_pmf >= 0 ? selected_pmf : light_pmf(s, cp.position, cp.shading_normal, sel);
            const float lpdf = env_image                        ? environment_image_pdf(s.img, direction, true) * sel_pmf
                               : nonzero3(lp.geometric_normal) ? sel_pmf * geometry_pdf
                                                               : 0.0f;
            bool ok;
            const V4 bsdf_pdf = represented_pdf<F == 3 ? 0 : F>(cbsdf, cframe, cp.position, previous, env_image,
                                                                env_image ? direction : lp.position, ok);
            weight_ok = ok && hero_weight(direct_density, value, v4(lpdf), bsdf_pdf, contribution);
        }
        // visible(): offset both endpoints (shaders/packet_transport.h:377-446)
        const V3 seg = lp.position - cp.position;
        if (!zero3(seg)) {
            const V3 so = offset_point(cp.position, cp.error, cp.geometric_normal, seg);
            const V3 st = offset_point(lp.position, lp.error, lp.geometric_normal, -seg);
            const V3 sd = st - so;
            shadow = true;
            sh_o = make_float4(so.x, so.y, so.z, kOneMinusEps);
            sh_d = make_float4(sd.x, sd.y, sd.z, __uint_as_float(path));
            sh_t = make_float4(st.x, st.y, st.z, 0);
            sh_c = weight_ok ? to_float4(contribution) : make_float4(__int_as_float(0x7fffffff), 0, 0, 0);
        }
    }
    if (status != 0) {
        ident.w = set_status(ident.w, status) | F_COMPLETE;
        pool.ident(path) = ident;
        shadow = false;
    }
}
// nee_path of the paths of family F with a request; the segments are queued for the shadow
// kernel.
template <int F, int Block = 128, bool Img = true>
__global__ void __launch_bounds__(Block, 512 / Block) k_nee(const __grid_constant__ DeviceScene s,
                                                            const __grid_constant__ WaveParams p, PathPool pool, int in,
                                                            u32 event_index) {
    u32 *event = pool.event(in);
    const u32 count = event[kNeeCount + F];
    const u32 *queue = pool.nee_queue + size_t(F) * pool.bin_capacity;
    const u32 stride = gridDim.x * blockDim.x;
    const u32 trips = (count + stride - 1) / stride;
    for (u32 trip = 0; trip < trips; ++trip) {
        const u32 i = trip * stride + blockIdx.x * blockDim.x + threadIdx.x;
        bool shadow = false;
        float4 sh_o = make_float4(0, 0, 0, 0), sh_d = sh_o, sh_c = sh_o, sh_t = sh_o;
        const bool active = i < count;
        nee_path<F, Img, true>(s, p, pool, in, event_index, active, active ? queue[i] : 0, shadow, sh_o, sh_d, sh_c, sh_t);
        const u32 sslot = warp_append(event + kShadowCount, shadow);
        if (shadow) {
            pool.sh_o[sslot] = sh_o;
            pool.sh_d[sslot] = sh_d;
            pool.sh_c[sslot] = sh_c;
            if (pool.sh_t)
                pool.sh_t[sslot] = sh_t;
        }
    }
}

// visible() through pass-through surfaces (shaders/packet_transport.h:393-445): nearest hits
// along the segment; an opaque one occludes, a pass-through one restarts the segment past it
// toward the target (at most boundary_limit + 1 walks).  Returns 0 with `occluded` set, or
// the failed sample's status (3 invalid hit, 2 invalid arithmetic, 4 boundary exhaustion).
template <bool Count, int Stack>
__device__ __noinline__ u32 pass_through_visible(const DeviceScene &s, V3 o, V3 d, float tmax, float4 target4,
                                                 bool &occluded, uint2 *stack, int stride, u32 boundary_limit,
                                                 u32 &nodes, u32 &tris, u32 &rays) {
    const V3 target = v3(target4.x, target4.y, target4.z);
    occluded = true;
    for (u32 crossings = 0; crossings <= boundary_limit; ++crossings) {
        Hit h;
        ++rays;
        if (!walk_closest<Count, Stack, true>(s, o, d, tmax, h, stack, stride, nodes, tris))
            return 3;
        if (h.prim == kNone) {
            occluded = false;
            return 0;
        }
        const u32 inst = s.tri_instance[h.prim];
        const DInstance &in = s.instances[inst];
        if (in.material >= s.material_count)
            return 3;
        if (!(in.resolve & kPassThrough))
            return 0;
        SurfacePoint pt;
        if (!hit_surface_point(s, h.prim, inst, s.tri_local[h.prim], h.b1, h.b2, pt))
            return 2;
        V3 next;
        if (!spawn_boundary(o, d, h.t, pt, normalize3(d), next))
            return 2;
        o = next;
        d = target - next;
    }
    return 4;
}

// What a light sample's visibility walk does to its path (visible(),
// shaders/packet_transport.h:377-446): the contribution where nothing occludes it, or the
// sample's failure.
template <bool Adjoint>
RP_DEV void shadow_result(const DeviceScene &s, const PathPool &pool, float *sgrad, const float4 &contribution, u32 path,
                          u32 failure, bool occluded) {
    if (!failure && occluded)
        return;
    uint4 ident = pool.ident(path);
    if (failure) {
        ident.w = set_status(ident.w, failure) | F_COMPLETE;
        pool.ident(path) = ident;
        return;
    }
    const float4 c = contribution;
    if (isnan(c.x)) {
        ident.w = set_status(ident.w, 2) | F_COMPLETE;
        pool.ident(path) = ident;
        return;
    }
    float4 r = pool.radiance(path);
    r.x += c.x;
    r.y += c.y;
    r.z += c.z;
    r.w += c.w;
    pool.radiance(path) = r;
    if (!finite_nonnegative4(from_float4(r))) {
        ident.w = set_status(ident.w, 2) | F_COMPLETE;
        pool.ident(path) = ident;
    } else if (Adjoint) {
        // replay: the light sample's gradient, over the history including its vertex
        adjoint_accumulate(s, pool, sgrad, pool.hist[path], from_float4(pool.lambda(path)), from_float4(c),
                           pool.adj_w[path]);
    }
}
struct ShadowRays {
    const DeviceScene &s;
    const PathPool &pool;
    u32 entry;

    template <class W> RP_DEV bool load(u32 i, W &w) {
        entry = i;
        const float4 o = pool.sh_o[i], d = pool.sh_d[i];
        w.start(s, v3(o.x, o.y, o.z), v3(d.x, d.y, d.z), o.w);
        return true;
    }
    template <class W> RP_DEV void finish(bool done, const W &w) {
        if (!done)
            return;
        const u32 path = __float_as_uint(pool.sh_d[entry].w);
        shadow_result<false>(s, pool, nullptr, pool.sh_c[entry], path, w.ok ? 0u : 3u, w.h.prim != kNone);
    }
    RP_DEV void flush() {}
};
// Visibility of the light samples, opaque surfaces; Resolve: the scene has pass-through
// instances, which shadow rays cross (pass_through_visible).
template <bool Count, int Block = kTraceBlock, bool Adjoint = false, int Stack = kStackDepth, bool Resolve = false,
          bool Stream = false>
__global__ void __launch_bounds__(Block, walk_blocks(Block, Stack, Stream))
    k_shadow(const __grid_constant__ DeviceScene s, PathPool pool, int in, u32 boundary_limit) {
    __shared__ uint2 stack[Stack * Block];
    extern __shared__ float sgrad[]; // adjoint only
    if (Adjoint)
        adjoint_begin(pool, sgrad);
    u32 *event = pool.event(in);
    const u32 count = event[kShadowCount];
    u32 nodes = 0, tris = 0, rays = 0;
    if constexpr (Stream) {
        static_assert(!Count && !Resolve && !Adjoint);
        ShadowRays io{s, pool, 0};
        walk_stream<Walker<true, Stack>>(s, count, event + kShadowNext, stack + threadIdx.x, Block, io);
    } else {
        for (u32 i = blockIdx.x * blockDim.x + threadIdx.x; i < count; i += gridDim.x * blockDim.x) {
            const float4 o = pool.sh_o[i], d = pool.sh_d[i];
            const u32 path = __float_as_uint(d.w);
            const u32 walks_before = rays;
            bool occluded;
            u32 failure = 0;
            if (Resolve) {
                failure = pass_through_visible<Count, Stack>(s, v3(o.x, o.y, o.z), v3(d.x, d.y, d.z), o.w, pool.sh_t[i],
                                                             occluded, stack + threadIdx.x, Block, boundary_limit, nodes,
                                                             tris, rays);
            } else {
                if (!walk_any<Count, Stack, false>(s, v3(o.x, o.y, o.z), v3(d.x, d.y, d.z), o.w, occluded,
                                                   stack + threadIdx.x, Block, nodes, tris))
                    failure = 3;
                ++rays;
            }
            if (Count && pool.lane_shadow)
                pool.lane_shadow[path] += rays - walks_before;
            shadow_result<Adjoint>(s, pool, sgrad, pool.sh_c[i], path, failure, occluded);
        }
    }
    if (Adjoint)
        adjoint_end(pool, sgrad);
    if (Count) {
        atomicAdd(pool.stats + 4, (unsigned long long)nodes);
        atomicAdd(pool.stats + 5, (unsigned long long)tris);
        atomicAdd(pool.stats + 3, (unsigned long long)rays);
    }
}

// Whole paths, one thread each: every event of a wave's paths, each the closest hit, the event,
// its light sample and that sample's visibility in turn, on the same path state as the wavefront
// kernels (so every lane's result is theirs).  A wave of few lanes is bound by the launches and
// the latencies of its events' kernels, not by their work: one launch runs it instead
// (whole_paths says when: its warps diverge over the families).  Scenes whose hits resolve before
// shading take the wavefront.
constexpr int kPathBlock = 64;
template <int Stack, bool Img>
__global__ void __launch_bounds__(kPathBlock, 6) k_paths(const __grid_constant__ DeviceScene s,
                                                         const __grid_constant__ WaveParams p, PathPool pool) {
    __shared__ uint2 stack[Stack * kPathBlock];
    for (u32 path = blockIdx.x * blockDim.x + threadIdx.x; path < p.lanes; path += gridDim.x * blockDim.x) {
        u32 unused = 0;
        for (u32 e = 0; e <= s.max_depth; ++e) {
            const int in = int(e & 1u);
            if (pool.ident(path).w & F_COMPLETE)
                break;
            const float4 o = pool.ray_o(in, path), d = pool.ray_d(in, path);
            Hit h;
            const bool hit_ok = walk_closest<false, Stack, false>(s, v3(o.x, o.y, o.z), v3(d.x, d.y, d.z),
                                                                  __int_as_float(0x7f800000), h, stack + threadIdx.x,
                                                                  kPathBlock, unused, unused);
            const u32 prim = hit_ok ? h.prim : kHitInvalid;
            const u32 family = !hit_ok || h.prim == kNone ? 3u : u32(__ldg(s.tri_family + h.prim));
            pool.hit(path) = make_float4(h.t, h.b1, h.b2, __uint_as_float(prim));
            bool keep = false, nee = false, shadow = false;
            float4 so, sd, sc, st;
            if (family == 0) {
                shade_path<0, false, Img, false>(s, p, pool, in, e, true, path, nullptr, keep, nee);
                if (nee)
                    nee_path<0, Img, false>(s, p, pool, in, e, true, path, shadow, so, sd, sc, st);
            } else if (family == 1) {
                shade_path<1, false, Img, false>(s, p, pool, in, e, true, path, nullptr, keep, nee);
                if (nee)
                    nee_path<1, Img, false>(s, p, pool, in, e, true, path, shadow, so, sd, sc, st);
            } else if (family == 2) {
                shade_path<2, false, Img, false>(s, p, pool, in, e, true, path, nullptr, keep, nee);
                if (nee)
                    nee_path<2, Img, false>(s, p, pool, in, e, true, path, shadow, so, sd, sc, st);
            } else {
                shade_path<3, false, Img, false>(s, p, pool, in, e, true, path, nullptr, keep, nee);
            }
            if (shadow) {
                bool occluded;
                const bool ok = walk_any<false, Stack, false>(s, v3(so.x, so.y, so.z), v3(sd.x, sd.y, sd.z), so.w,
                                                              occluded, stack + threadIdx.x, kPathBlock, unused, unused);
                shadow_result<false>(s, pool, nullptr, sc, path, ok ? 0u : 3u, occluded);
            }
            if (!keep)
                break;
        }
    }
}

// packet_pt_result (shaders/packet_pt_step.h:225-239): 80-byte packet result per lane.  The
// reserved words, which rypath leaves unread, carry the lane's closest-hit and any-hit walk
// counts in counting runs (zero otherwise).
struct PacketResult {
    u32 status, pixel, sample_low, sample_high, splat_count;
    float wavelengths[4], wavelength_pdfs[4], radiance[4];
    float filter_weight;
    u32 reserved[2];
};
// failed (null: not wanted; zero before): the complement of the first failed lane, [1] their
// number, so that the host need not read every lane's status (1.3 ms of 20 MB of lanes).
RP_DEV void count_failed(u32 *failed, u32 lane, u32 status) {
    if (failed && status) {
        atomicMax(failed, ~lane);
        atomicAdd(failed + 1, 1u);
    }
}
__global__ void k_results(PathPool pool, u32 lanes, float filter_weight, PacketResult *out, u32 *failed) {
    for (u32 lane = blockIdx.x * blockDim.x + threadIdx.x; lane < lanes; lane += gridDim.x * blockDim.x) {
        const uint4 id = pool.ident(lane);
        const float4 l = pool.lambda(lane), pdf = pool.lambda_pdf(lane), r = pool.radiance(lane);
        PacketResult res;
        res.status = (id.w & F_COMPLETE) ? get_status(id.w) : 2u;
        count_failed(failed, lane, res.status);
        res.pixel = id.x;
        res.sample_low = id.y;
        res.sample_high = id.z;
        res.splat_count = 0;
        res.wavelengths[0] = l.x;
        res.wavelengths[1] = l.y;
        res.wavelengths[2] = l.z;
        res.wavelengths[3] = l.w;
        res.wavelength_pdfs[0] = pdf.x;
        res.wavelength_pdfs[1] = pdf.y;
        res.wavelength_pdfs[2] = pdf.z;
        res.wavelength_pdfs[3] = pdf.w;
        res.radiance[0] = r.x;
        res.radiance[1] = r.y;
        res.radiance[2] = r.z;
        res.radiance[3] = r.w;
        res.filter_weight = filter_weight;
        res.reserved[0] = pool.lane_closest ? pool.lane_closest[lane] : 0u;
        res.reserved[1] = pool.lane_shadow ? pool.lane_shadow[lane] : 0u;
        out[lane] = res;
    }
}

// Device film pixel: FP64 Neumaier sums (src/packet_film.cpp:10-14, :198-265) plus second moments.
struct FilmPixel {
    double sum[3], correction[3];
    double weight_sum, weight_correction;
    double square[3];
    unsigned long long count;
    double compatibility_sum[3], compatibility_correction[3];
};
// A finite film clamp (on: max_component_value finite and positive).
struct FilmClamp {
    double exposure, max_component_value;
    bool on;
};
RP_DEV void add_compensated(double value, double &sum, double &correction) {
    const double next = __dadd_rn(sum, value);
    correction = __dadd_rn(correction, fabs(sum) >= fabs(value) ? __dadd_rn(__dsub_rn(sum, next), value)
                                                                  : __dadd_rn(__dsub_rn(value, next), sum));
    sum = next;
}
// packet_sensor_xyz (src/packet_film.cpp:102-114) of one lane added to its pixel; false when
// the lane failed (a failed lane fails its batch).
// clamp_sensor + add_xyz into the compatibility planes (src/packet_film.cpp:39-56, :217-220)
RP_DEV void film_add_compatibility(const double (&xyz)[3], double weight, const FilmClamp &c, FilmPixel &f) {
    double v[3];
#pragma unroll
    for (int k = 0; k < 3; ++k)
        v[k] = __dmul_rn(xyz[k], c.exposure);
    double maximum = v[0];
    if (v[1] > maximum)
        maximum = v[1];
    if (v[2] > maximum)
        maximum = v[2];
    if (maximum > c.max_component_value) {
        const double scale = __ddiv_rn(c.max_component_value, maximum);
#pragma unroll
        for (int k = 0; k < 3; ++k)
            v[k] = __dmul_rn(v[k], scale);
    }
#pragma unroll
    for (int k = 0; k < 3; ++k)
        add_compensated(__dmul_rn(v[k], weight), f.compatibility_sum[k], f.compatibility_correction[k]);
}
RP_DEV bool film_add_lane(const PathPool &pool, u32 lane, const double *cie, double weight, const FilmClamp &clamp,
                          FilmPixel &f) {
    const uint4 id = pool.ident(lane);
    const u32 status = (id.w & F_COMPLETE) ? get_status(id.w) : 2u;
    if (status != 0)
        return false;
    const float4 l4 = pool.lambda(lane), p4 = pool.lambda_pdf(lane), r4 = pool.radiance(lane);
    const float lam[4] = {l4.x, l4.y, l4.z, l4.w}, pdf[4] = {p4.x, p4.y, p4.z, p4.w}, rad[4] = {r4.x, r4.y, r4.z, r4.w};
    double xyz[3] = {0, 0, 0};
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        if (pdf[k] == 0)
            continue;
        const float w = lam[k];
        if (!(w >= 360 && w <= 830))
            continue;
        const u32 row = u32(round(double(w)) - 360.0);
        const double weight = __ddiv_rn(__ddiv_rn(double(rad[k]), double(pdf[k])), 4.0);
#pragma unroll
        for (int c = 0; c < 3; ++c)
            xyz[c] = __dadd_rn(xyz[c], __dmul_rn(weight, __ldg(cie + 3 * row + c)));
    }
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        const double v = __dmul_rn(xyz[c], weight); // add_xyz (src/packet_film.cpp:46-56)
        add_compensated(v, f.sum[c], f.correction[c]);
        f.square[c] = __dadd_rn(f.square[c], __dmul_rn(v, v));
    }
    if (clamp.on)
        film_add_compatibility(xyz, weight, clamp, f);
    add_compensated(weight, f.weight_sum, f.weight_correction);
    ++f.count;
    return true;
}
// Failed lanes of a wave (counters[3]), for passes that produce no film.  counters[3] is
// cleared with the wave's counters, so callers accumulate it per wave.
__global__ void k_count_failures(PathPool pool, u32 lanes) {
    for (u32 lane = blockIdx.x * blockDim.x + threadIdx.x; lane < lanes; lane += gridDim.x * blockDim.x) {
        const u32 w = pool.ident(lane).w;
        if (!(w & F_COMPLETE) || get_status(w) != 0)
            atomicAdd(pool.counters + 3, 1u);
    }
}
// The DrawTables of the draw blocks [first, first + blocks), for the hero transport [133, 133 +
// blocks), and block 0: `tables` in all.
RP_DEV u32 draw_block_of(u32 slot, u32 first, u32 blocks, u32 tables) {
    return slot == tables - 1 ? 0 : slot < blocks ? first + slot : 133 + (slot - blocks);
}
__global__ void k_draw_tables(SobolTables sobol, unsigned short *prefix, uint4 *bytes, u32 *hash, u32 first, u32 blocks,
                              u32 tables, u32 seed) {
    const u32 prefixes = tables * 4 * kOwenPrefixEntries, products = tables * kIndexBytes * 256;
    const u32 stride = gridDim.x * blockDim.x, begin = blockIdx.x * blockDim.x + threadIdx.x;
    for (u32 e = begin; e < prefixes; e += stride) {
        const u32 slot = e / (4 * kOwenPrefixEntries), k = (e / kOwenPrefixEntries) & 3u;
        const u32 block = draw_block_of(slot, first, blocks, tables);
        const u32 h = sobol_dimension_hash(4 * block + k, seed);
        prefix[e] = (unsigned short)owen_prefix_rounds(e % kOwenPrefixEntries, h);
        if (e % kOwenPrefixEntries == 0)
            hash[4 * slot + k] = h;
    }
    for (u32 e = begin; e < products; e += stride) {
        const u32 slot = e / (kIndexBytes * 256), byte = (e >> 8) % kIndexBytes, value = e & 0xffu;
        const u32 block = draw_block_of(slot, first, blocks, tables);
        u32 v[4] = {0, 0, 0, 0};
        for (u32 bit = 0; bit < 8 && 8 * byte + bit < kSobolMatrix; ++bit)
            if (value >> bit & 1u)
                for (u32 k = 0; k < 4; ++k)
                    if (4 * block + k < 1024u)
                        v[k] ^= __ldg(sobol.directions + (4 * block + k) * kSobolMatrix + 8 * byte + bit);
        bytes[e] = make_uint4(v[0], v[1], v[2], v[3]);
    }
}

// Every sample of a wave reduced per pixel in canonical (absolute sample, pixel) order.
__global__ void k_film(PathPool pool, u32 pixel_count, u32 samples, const double *cie, double weight, FilmClamp clamp,
                       FilmPixel *film) {
    for (u32 px = blockIdx.x * blockDim.x + threadIdx.x; px < pixel_count; px += gridDim.x * blockDim.x) {
        FilmPixel f = film[px];
        for (u32 si = 0; si < samples; ++si)
            if (!film_add_lane(pool, si * pixel_count + px, cie, weight, clamp, f))
                atomicAdd(pool.counters + 3, 1u);
        film[px] = f;
    }
}

// The frame sensor of a packet lane (shaders/frame_sensor.h:33-52): raw XYZ of one camera
// sample, sum over the valid wavelength lanes of the matching functions at the nearest
// nanometre times radiance / pdf / 4, in binary32 (the filter weight cancels against its own
// normalisation).  A failed or inconsistent lane (status, identity, a companion terminated
// beside a surviving one, a non-finite value) writes zero and counts a failure.
__global__ void k_frame_packet(PathPool pool, u32 pixel_count, u32 pixel_begin, u32 sample_low, u32 sample_high,
                               const double *cie, float *xyz, u32 *failures) {
    for (u32 px = blockIdx.x * blockDim.x + threadIdx.x; px < pixel_count; px += gridDim.x * blockDim.x) {
        const uint4 id = pool.ident(px);
        bool valid = (id.w & F_COMPLETE) && get_status(id.w) == 0 && id.x == pixel_begin + px && id.y == sample_low &&
                     id.z == sample_high;
        const float4 l4 = pool.lambda(px), p4 = pool.lambda_pdf(px), r4 = pool.radiance(px);
        const float lam[4] = {l4.x, l4.y, l4.z, l4.w}, pdf[4] = {p4.x, p4.y, p4.z, p4.w}, rad[4] = {r4.x, r4.y, r4.z, r4.w};
        bool secondary = false, terminated = false;
        float v[3] = {0, 0, 0};
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const bool good = lam[k] >= 360 && lam[k] <= 830 && isfinite(pdf[k]) && pdf[k] >= 0 && (k != 0 || pdf[k] > 0) &&
                              isfinite(rad[k]) && rad[k] >= 0;
            valid = valid && good;
            if (k > 0) {
                secondary = secondary || pdf[k] > 0;
                terminated = terminated || pdf[k] == 0;
            }
            if (good && pdf[k] > 0) {
                const u32 row = u32(floorf(lam[k] + .5f) - 360.f);
                const float w = rad[k] / pdf[k] / 4.f;
#pragma unroll
                for (int c = 0; c < 3; ++c)
                    v[c] = v[c] + float(__ldg(cie + 3 * row + c)) * w;
            }
        }
        valid = valid && !(secondary && terminated) && isfinite(v[0]) && isfinite(v[1]) && isfinite(v[2]);
        if (!valid) {
            v[0] = v[1] = v[2] = 0;
            atomicAdd(failures, 1u);
        }
        xyz[3 * size_t(px)] = v[0];
        xyz[3 * size_t(px) + 1] = v[1];
        xyz[3 * size_t(px) + 2] = v[2];
    }
}

} // namespace rp
