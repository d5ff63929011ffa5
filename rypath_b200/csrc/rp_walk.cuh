// Streaming walks of the wide tree: a warp keeps its lanes on rays of its own and hands a lane
// the next ray of the launch when its ray ends, instead of waiting for the longest ray of 32.
//
// The walk is bound by instruction issue, and rays of one warp end after very different
// numbers of node visits (the longest of 32 takes about three times the mean) and reach leaves
// at different visits.  Three things keep the lanes of an issued instruction busy: lanes whose
// rays ended are refilled once kRefill of them wait; node visits and triangle tests
// are separate steps of the warp, and a lane whose visit found leaves waits for its tests
// until kLeafLanes lanes have some (or no lane can visit a node); results leave through
// per-warp queues in shared memory that append 32 entries at a time.  A ray's hits do not
// depend on any of this: the visits of one ray and its tests are those of walk_closest and
// walk_any, in the same order.  Mixed scene, event 1: 9.5 of 32 lanes active an instruction
// before, 12.7 so; 1080p, 16 spp 83.9 -> 81.6 ms.  Refill / leaf thresholds 4/8, 16/12, 8/14 and 14/14 were slower
// than 12/10.
#pragma once

#include "rp_scene.cuh"

namespace rp {

constexpr u32 kRefill = 12;     // waiting lanes that start a refill
constexpr u32 kLeafLanes = 10; // lanes with leaves that start a triangle step

// One ray's walk, advanced a node visit or a triangle test at a time.  Any: occlusion in
// (0, h.t); else closest hit, minimising (t, primitive id) over (0, tmax).
template <bool Any, int Stack> struct Walker {
    WalkRay r;
    WideRay wr;
    Hit h;       // closest: the best hit so far, t its limit; any: t = tmax, prim set once occluded
    float tmax;
    u32 order;
    u32 node;    // next node to visit, kNone: none left
    u32 tri_base, leaves; // untested leaves of the last visit: hit bits, leaf mask << 8
    u32 visits;  // bounds the walk: a node is visited at most once
    int sp;
    bool ok;     // false: the stack overflowed (a failed query)

    RP_DEV bool has_leaves() const { return (leaves & 0xffu) != 0; }
    RP_DEV bool ended() const { return node == kNone && !has_leaves(); }
    RP_DEV void skip() {
        node = kNone;
        leaves = 0;
        ok = true;
        visits = 0;
    }
    RP_DEV void start(const DeviceScene &s, V3 o, V3 d, float limit) {
        skip();
        h.t = tmax = limit;
        h.b1 = h.b2 = 0;
        h.prim = kNone;
        sp = 0;
        r = walk_ray(o, d);
        wr = wide_ray(d);
        order = (d.x < 0 ? 1u : 0u) | (d.y < 0 ? 2u : 0u) | (d.z < 0 ? 4u : 0u);
        if (s.prim_count > 1) {
            node = 0;
        } else if (s.prim_count == 1) {
            tri_base = 0;
            leaves = 1u | (1u << 8);
        }
    }
    RP_DEV void visit(const DeviceScene &s, uint2 *stack, int stride) {
        const WNode *np = s.wnodes + node;
        const float4 origin = __ldg(&np->origin);
        const uint4 links = __ldg(&np->links);
        u32 inner, hit_leaves;
        wide_children(np, origin, links, r.o, wr, h.t, order, inner, hit_leaves);
        tri_base = links.y;
        leaves = hit_leaves | (links.z << 8);
        u32 base = links.x, group_mask = __float_as_uint(origin.w) >> 24;
        if (!inner) {
            if (sp == 0) {
                node = kNone;
                return;
            }
            --sp;
            const uint2 e = stack[sp * stride];
            base = e.x;
            group_mask = e.y >> 8;
            inner = e.y & 0xffu;
        }
        const u32 b = __ffs(inner) - 1;
        inner &= inner - 1;
        const u32 slot = b ^ order;
        node = base + __popc(group_mask & ((1u << slot) - 1));
        if (inner) {
            if (sp >= Stack) {
                fail();
                return;
            }
            stack[sp * stride] = make_uint2(base, (group_mask << 8) | inner);
            ++sp;
        }
        if (visits++ >= s.wnode_count) // no valid tree has a node more to visit
            fail();
    }
    RP_DEV void fail() {
        ok = false;
        node = kNone;
        leaves = 0;
    }
    RP_DEV void test(const DeviceScene &s) {
        const u32 k = __ffs(leaves) - 1;
        const u32 index = tri_base + __popc((leaves >> 8) & ((1u << k) - 1));
        leaves &= ~(1u << k);
        u32 unused = 0;
        if constexpr (Any) {
            if (any_leaf<false, false>(s, r, tmax, index, unused)) {
                h.prim = 0;
                node = kNone;
                leaves = 0;
            }
        } else {
            closest_leaf<false, false>(s, r, tmax, h, index, unused);
        }
    }
};

// Rays [0, count) of a launch, in chunks that the warps take from `cursor` (zero at launch).
// Io::load(i, walker) starts ray i (false: nothing to do); Io::finish(done, walker) takes
// the results of the lanes with `done`, called by the whole warp; Io::flush() ends the launch.
template <class W, class Io>
RP_DEV void walk_stream(const DeviceScene &s, u32 count, u32 *cursor, uint2 *stack, int stride, Io &io) {
    const u32 lane = threadIdx.x & 31;
    // several chunks a warp for balance, whole warps of rays, few atomics on the cursor
    const u32 warps = (gridDim.x * blockDim.x) >> 5;
    const u32 chunk = min(256u, max(32u, (count / (4 * warps)) & ~31u));
    W w;
    w.skip();
    bool active = false, drained = false;
    u32 next = 0, end = 0; // the warp's chunk
    for (;;) {
        u32 idle = __ballot_sync(0xffffffffu, !active);
        if (!drained && next == end) {
            if (lane == 0)
                next = atomicAdd(cursor, chunk);
            next = __shfl_sync(0xffffffffu, next, 0);
            end = min(next + chunk, count);
            if (next >= count) {
                drained = true;
                next = end;
            }
        }
        if (next < end) {
            const u32 take = min(u32(__popc(idle)), end - next);
            const u32 rank = __popc(idle & ((1u << lane) - 1));
            if (!active && rank < take)
                active = io.load(next + rank, w);
            next += take;
            idle = __ballot_sync(0xffffffffu, !active);
        }
        if (idle == 0xffffffffu) {
            if (drained)
                break;
            continue;
        }
        for (;;) {
            const u32 leaf = __ballot_sync(0xffffffffu, active && w.has_leaves());
            const u32 open = __ballot_sync(0xffffffffu, active && !w.has_leaves() && w.node != kNone);
            const u32 waiting = 32 - __popc(leaf | open);
            if (waiting == 32 || (!drained && waiting >= kRefill))
                break;
            if (__popc(leaf) >= kLeafLanes || !open) {
                if (leaf >> lane & 1u)
                    w.test(s);
            } else if (open >> lane & 1u) {
                w.visit(s, stack, stride);
            }
        }
        const bool done = active && w.ended();
        io.finish(done, w);
        if (done)
            active = false;
    }
    io.flush();
}

// A warp's staged appends to four device queues: entries gather in shared memory and leave 32
// at a time, one atomic and one coalesced store for each 32.
constexpr u32 kStageEntries = 64;
struct StagedAppend {
    u32 *stage;   // this warp's 4 x kStageEntries words
    u32 counts;   // entries of each queue, a byte each

    RP_DEV void push(u32 q, bool want, u32 value, u32 *counter, u32 *queue) {
        const u32 ballot = __ballot_sync(0xffffffffu, want);
        if (!ballot)
            return;
        const u32 lane = threadIdx.x & 31, shift = 8 * q;
        u32 *e = stage + q * kStageEntries;
        const u32 have = (counts >> shift) & 0xffu, n = __popc(ballot);
        if (want)
            e[have + __popc(ballot & ((1u << lane) - 1))] = value;
        __syncwarp();
        if (have + n < 32) {
            counts += n << shift;
            return;
        }
        u32 base = 0;
        if (lane == 0)
            base = atomicAdd(counter, 32u);
        base = __shfl_sync(0xffffffffu, base, 0);
        const u32 out = e[lane], rest = e[32 + lane];
        queue[base + lane] = out;
        __syncwarp();
        e[lane] = rest;
        __syncwarp();
        counts += (n - 32) << shift;
    }
    RP_DEV void flush(u32 q, u32 *counter, u32 *queue) {
        const u32 lane = threadIdx.x & 31, have = (counts >> (8 * q)) & 0xffu;
        if (!have)
            return;
        u32 base = 0;
        if (lane == 0)
            base = atomicAdd(counter, have);
        base = __shfl_sync(0xffffffffu, base, 0);
        if (lane < have)
            queue[base + lane] = stage[q * kStageEntries + lane];
        __syncwarp();
    }
};

} // namespace rp
