// Software traversal over the reference's own two-level binary trees (renderer/shaders/trace_units.wgsl:44-135):
// the top tree over the units' world boxes, each unit's mesh tree in its model space, one loop over both levels.
// It is the pass's walk (faster on B200 than the wide-BVH walk of wide_bvh.cuh, which TRT_RENDER_WIDE selects).
#pragma once
#include "device_common.cuh"

namespace trt {

struct Hit { float t; uint32_t tri; float u, v; uint32_t inst, part; };

// Three-input minimum and maximum (one instruction each on sm_100; exact, like two fminf / fmaxf).
__device__ __forceinline__ float max3f(float a, float b, float c) {
    float r;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}
__device__ __forceinline__ float min3f(float a, float b, float c) {
    float r;
    asm("min.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}

// pathtrace.wgsl:732-739 ray_aabb over a node record's two halves, as a predicate and the entry distance (min and max are
// exact, so grouping them three at a time rounds nothing).
__device__ __forceinline__ bool box_hit(V3 o, V3 inv_d, const uint4& a, const uint4& b, float tmax, float& tn) {
    const float x0 = (bf(a.x) - o.x) * inv_d.x, y0 = (bf(a.y) - o.y) * inv_d.y, z0 = (bf(a.z) - o.z) * inv_d.z;
    const float x1 = (bf(b.x) - o.x) * inv_d.x, y1 = (bf(b.y) - o.y) * inv_d.y, z1 = (bf(b.z) - o.z) * inv_d.z;
    tn = max3f(fminf(x0, x1), fminf(y0, y1), fmaxf(fminf(z0, z1), 0.0f));
    const float tf = min3f(fmaxf(x0, x1), fmaxf(y0, y1), fminf(fmaxf(z0, z1), tmax));
    return tn <= tf;
}

// pathtrace.wgsl:742-761 intersect_tri (Moller-Trumbore on the leaf's v0, e1, e2), t = INF for none.
__device__ __forceinline__ float3 intersect_tri(const DScene& S, V3 o, V3 d, uint32_t i, float tmax) {
    float4 a = __ldg(S.leaves + 3ull * i), b = __ldg(S.leaves + 3ull * i + 1), c = __ldg(S.leaves + 3ull * i + 2);
    V3 v0 = xyz(a), e1 = xyz(b), e2 = xyz(c);
    V3 pv = cross(d, e2);
    float det = dot(e1, pv);
    if (fabsf(det) < 1e-12f) return make_float3(INF, 0.0f, 0.0f);
    float inv = 1.0f / det;
    V3 tv = o - v0;
    float u = dot(tv, pv) * inv;
    if (u < 0.0f || u > 1.0f) return make_float3(INF, 0.0f, 0.0f);
    V3 qv = cross(tv, e1);
    float v = dot(d, qv) * inv;
    if (v < 0.0f || u + v > 1.0f) return make_float3(INF, 0.0f, 0.0f);
    float t = dot(e2, qv) * inv;
    if (t <= 0.0f || t >= tmax) return make_float3(INF, 0.0f, 0.0f);
    return make_float3(t, u, v);
}

// pathtrace.wgsl:661 proc_dir: world -> a record's model space by its normal rows.
__device__ __forceinline__ V3 proc_dir(const float4& n0, const float4& n1, const float4& n2, V3 d) {
    return xyz(n0) * d.x + xyz(n1) * d.y + xyz(n2) * d.z;
}
__device__ __forceinline__ V3 safe_inv(V3 d) {
    V3 s = {fabsf(d.x) < 1e-20f ? 1e-20f : d.x, fabsf(d.y) < 1e-20f ? 1e-20f : d.y, fabsf(d.z) < 1e-20f ? 1e-20f : d.z};
    return V3{1.0f / s.x, 1.0f / s.y, 1.0f / s.z};
}

struct WalkCount { uint32_t nodes, tris, units; };

// The loop guard (renderer/src/gpu.rs:1214-1285 guard_loops): a walk that has not ended after this many nodes stops,
// sets *guard and returns what it has; the render then reports an error instead of hanging on trees that are not
// trees.
constexpr uint32_t WALK_GUARD = 1u << 20;

// trace_units.wgsl:44-135, with a 64-entry stack of its own. Returns the hit (tri MISS for none).
//
// The loop is split in two (Aila and Laine's "while-while"): interior nodes in an inner loop until a leaf, then the
// leaf (a unit's record, or a mesh's triangles). What bounds it is issue, above all of the half-rate integer and
// min / max pipe, at 8-10 of 32 lanes a warp instruction: ncu on a 512 x 512 town, depth 1, had 65-69 % of issue slots
// and 52-57 % of that pipe busy, DRAM and L2 below 10 %, and neither fewer loads a step, nor prefetching the stacked
// nodes, nor packed two-lane arithmetic moved the time. So the step is short: a child's link and count come with its
// box (the node is not read again when the walk descends into it), the box tests answer with predicates, a pair's four
// loads share one address, indices are checked in 32 bits, and a stack entry is a node's index, read again when it is
// popped (keeping the links on the stack took five more instructions a step than the two loads at a pop). Warp
// instructions of that depth: 82.2 -> 75.1 M closest, 139.6 -> 125.4 M shadow; the city frame (720p, 1 spp, depth 4)
// 4.89 -> 4.49 ms, the town (512 x 512, 16 spp) 18.34 -> 16.90 ms. With the loop unsplit (each node a round of one
// loop) the walks of the camera's rays are no faster (4.56 ms); 7 or 9 blocks an SM instead of 8: 4.55 and 4.60 ms.
template <bool COUNT>
__device__ __forceinline__ Hit trace_binary(const DScene& S, const Sections& X, uint32_t top, uint32_t n_units, V3 o, V3 d,
                                            float tmax, uint32_t mode, WalkCount* wc, bool* guard) {
    Hit hit{tmax, MISS, 0.0f, 0.0f, NO_INST, 0u};
    if (n_units == 0) return hit;
    if (top >= S.n_nodes) { *guard = true; return hit; }
    V3 inv_d = safe_inv(d);
    // The buffers' ends in 32 bits, as the indices are: the last node (a pair of children starts before it), the
    // triangles, the tables.
    const uint32_t last_node = (uint32_t)min((unsigned long long)S.n_nodes - 1ull, 0xffffffffull);
    const uint32_t tris_end = (uint32_t)min((unsigned long long)S.n_tris, 0xffffffffull);
    const uint32_t tables_end = (uint32_t)min((unsigned long long)S.n_table_vec4, 0xffffffffull);
    // The node the walk is at: `count` 0, an interior node, `at` its left child's index; else a leaf, `at` the first
    // of its `count` items.
    uint32_t at, count;
    {
        const uint4* q = S.nodes + 2ull * top;
        const uint4 a = __ldg(q), b = __ldg(q + 1);
        float t;
        if (COUNT) wc->nodes++;
        if (!box_hit(o, inv_d, a, b, hit.t, t)) return hit;
        if (COUNT) wc->nodes++;
        count = b.w;
        at = count == 0 ? a.w + top : a.w;
    }
    uint32_t stack[64];
    uint32_t sp = 0, rec = NO_INST;
    constexpr uint32_t NO_BASE = 0xffffffffu;  // (base outside a unit: no height of the stack)
    uint32_t off = top, first = 0, base = NO_BASE;
    V3 ro = o, rd = d, rinv = inv_d;
    // Out of a unit whose subtree is done, then the next node (false: the walk is over).
    auto pop = [&]() -> bool {
        if (sp == base) {
            rec = NO_INST;
            base = NO_BASE;
            ro = o; rd = d; rinv = inv_d;
            off = top;
        }
        if (sp == 0) return false;
        const uint32_t* q = reinterpret_cast<const uint32_t*>(S.nodes + 2ull * stack[--sp]);
        if (COUNT) wc->nodes++;
        at = __ldg(q + 3);
        count = __ldg(q + 7);
        if (count == 0) at += off;
        return true;
    };
    uint32_t iter = 0;
    for (;;) {
        // (Every index a walk follows is checked: a bad tree ends the walk with the guard set, never a fault.)
        bool over = false;
        while (count == 0) {
            if (iter++ >= WALK_GUARD || at >= last_node) { *guard = true; return hit; }
            const uint4* q = S.nodes + 2ull * at;
            const uint4 l0 = __ldg(q), l1 = __ldg(q + 1), r0 = __ldg(q + 2), r1 = __ldg(q + 3);
            if (COUNT) wc->nodes += 2;
            float tl, tr;
            const bool hl = box_hit(ro, rinv, l0, l1, hit.t, tl), hr = box_hit(ro, rinv, r0, r1, hit.t, tr);
            if (hl || hr) {
                const bool swap = hr && (!hl || tr < tl);
                const uint32_t link = swap ? r0.w : l0.w;
                count = swap ? r1.w : l1.w;
                if (COUNT) wc->nodes++;
                if (hl && hr && sp < 64) stack[sp++] = swap ? at : at + 1u;
                at = count == 0 ? link + off : link;
            } else if (!pop()) {
                over = true;
                break;
            }
        }
        if (over) break;
        if (iter++ >= WALK_GUARD) { *guard = true; return hit; }
        if (rec == NO_INST) {
            uint32_t b = X.t_instances + at * 10u;
            if (tables_end < 10u || b > tables_end - 10u) { *guard = true; return hit; }
            const uint4* u = S.tables + b;
            const float4* uf = reinterpret_cast<const float4*>(u);
            const float4 n1 = __ldg(uf + 4);
            uint32_t ubits = bu(n1.w);
            if (COUNT) wc->units++;
            if (mode != TRACE_SHADOW || (ubits & UNIT_SHADOW) != 0) {
                const float4 n0 = __ldg(uf + 3), n2 = __ldg(uf + 5);
                rec = at;
                ro = o - V3{__ldg(&uf[0].w), __ldg(&uf[1].w), __ldg(&uf[2].w)};
                first = __ldg(&u[6].x);
                if ((ubits & UNIT_SHIFTED) == 0) {
                    ro = proc_dir(n0, n1, n2, ro);
                    rd = proc_dir(n0, n1, n2, d);
                    rinv = safe_inv(rd);
                }
                off = bu(n0.w);
                base = sp;
                if (off > last_node) { *guard = true; return hit; }
                const uint32_t* q = reinterpret_cast<const uint32_t*>(S.nodes + 2ull * off);
                at = __ldg(q + 3);
                count = __ldg(q + 7);
                if (COUNT) wc->nodes++;
                if (count == 0) at += off;
                continue;
            }
        } else {
            for (uint32_t k = 0; k < count; ++k) {
                uint32_t ti = first + at + k;
                if (ti >= tris_end) { *guard = true; return hit; }
                if (COUNT) wc->tris++;
                float3 x = intersect_tri(S, ro, rd, ti, hit.t);
                if (x.x < hit.t) {
                    uint32_t part = bu(__ldg(S.leaves + 3ull * ti).w);
                    hit = Hit{x.x, ti, x.y, x.z, rec, part};
                    if (mode != TRACE_CLOSEST) return hit;
                }
            }
        }
        if (!pop()) break;
    }
    return hit;
}

__device__ __forceinline__ uint32_t end32(unsigned long long n) { return (uint32_t)min(n, 0xffffffffull); }

// The same walk over a stream of rays, for waves whose rays go many ways through deep trees: a warp keeps its lanes in
// work. trace_binary's lanes wait for each other twice: those at a leaf until the last of the warp has left the inner
// loop, and those whose ray has ended until the warp's longest ray has; 7-9 of 32 lanes are left a warp instruction.
// Here the warp runs, each round, the phase that most of its lanes wait for (a few interior steps, or entering a
// unit, or a leaf's triangles), and when STREAM_REFILL lanes are idle these take the next rays together. Neither half
// gives anything alone (refilling trace_binary's lanes made it 6 % slower, the vote without refills 0 %), and a round
// for both leaf kinds at once or an inner loop that runs until few lanes are left in it were slower too (town below:
// 15.95-16.6 ms). A town's second depth (640 x 512, 1 spp): 7.6 -> 13.4 lanes and 175 -> 140 M warp instructions for its
// shadow rays, 8.8 -> 13.7 and 101 -> 92 M closest; the more rays a warp gets, the better (34 of them, no gain; 400,
// 30 % by a count of the phases), and short walks lose (the rounds cost a quarter more thread instructions): the caller
// chooses. The town at 512 x 512, 16 spp, 16.85 -> 15.36 ms; the city frame (720p, 1 spp) 4.46 -> 4.27. STREAM_STEPS /
// STREAM_REFILL 3 / 12: 15.69, 4 / 16: 15.63, 6 / 16: 15.66, 2 / 8: 16.14 (before the other ballots were put off).
//
// n rays, handed out by `counter`. load(i, ray, o, d, t, mode) fetches the i-th and names it; its scene is `one`, or, where
// Lane::ON, what load has bound `view` to; hit(ray, x, tri, rec) takes a nearer hit (t, u, v) and says whether the ray is
// done; done(ray) ends one, unless hit() set it to NO_RAY. What a ray meets, and in which order, is trace_binary's, and so
// are the checks of every index and WALK_GUARD (a ray each).
constexpr uint32_t NO_RAY = 0xffffffffu;
constexpr int STREAM_STEPS = 4, STREAM_REFILL = 16;
template <class Lane, class Load, class Take, class Done>
__device__ __forceinline__ void trace_stream(const DScene& one, uint32_t one_instances, uint32_t one_top, uint32_t one_units,
                                             Lane& view, uint32_t* counter, uint32_t n, Load load, Take hit, Done done,
                                             unsigned long long& guard_trips) {
    constexpr unsigned ALL = 0xffffffffu;
    constexpr uint32_t IDLE = 0xffffffffu, NO_BASE = 0xffffffffu;
    const uint32_t one_last = end32(one.n_nodes - 1ull);
    const uint32_t one_tris = end32(one.n_tris);
    const uint32_t one_tables = end32(one.n_table_vec4);
    auto nodes = [&]() -> const uint4* { if constexpr (Lane::ON) return view.nodes; else return one.nodes; };
    auto last_node = [&]() -> uint32_t { if constexpr (Lane::ON) return view.last; else return one_last; };
    auto top_of = [&]() -> uint32_t { if constexpr (Lane::ON) return view.top(); else return one_top; };
    const uint32_t lane = threadIdx.x & 31u;
    V3 o{0.0f, 0.0f, 0.0f}, d = o, inv_d = o, ro = o, rd = o, rinv = o;
    float t = 0.0f;
    // `count` IDLE: the lane has no ray, or its ray has ended (`ray`: it is not handed on yet). A leaf's count may be any
    // number but zero (it counts triangles up to the buffer's end, of a unit it says nothing), so a node's is taken as
    // IDLE - 1 at most. (0.25 % of the city still; a mark of its own kept the shadow walk's registers past 56, 0.6 %.)
    uint32_t ray = NO_RAY, mode = 0, at = 0, count = IDLE, off = 0, first = 0, rec = NO_INST, iter = 0;
    uint32_t stack[64];
    uint32_t sp = 0, base = NO_BASE;
    auto trip = [&]() { guard_trips++; count = IDLE; };
    auto pop = [&]() {
        if (sp == base) {
            rec = NO_INST;
            base = NO_BASE;
            ro = o; rd = d; rinv = inv_d;
            off = top_of();
        }
        if (sp == 0) { count = IDLE; return; }
        const uint32_t* q = reinterpret_cast<const uint32_t*>(nodes() + 2ull * stack[--sp]);
        at = __ldg(q + 3);
        count = min(__ldg(q + 7), IDLE - 1u);
        if (count == 0) at += off;
    };
    bool more = n != 0;
    for (;;) {
        const unsigned busy = __ballot_sync(ALL, count != IDLE);
        const int n_busy = __popc(busy);
        if (more && n_busy <= 32 - STREAM_REFILL) {
            const uint32_t want = 32u - (uint32_t)n_busy;
            uint32_t b = 0;
            if (lane == 0) b = atomicAdd(counter, want);
            b = __shfl_sync(ALL, b, 0);
            more = b < n && n - b > want;
            if (count == IDLE) {
                if (ray != NO_RAY) done(ray);
                ray = NO_RAY;
                const uint32_t i = b + (uint32_t)__popc(~busy & ((1u << lane) - 1u));
                if (b < n && i < n) {
                    load(i, ray, o, d, t, mode);
                    inv_d = safe_inv(d);
                    ro = o; rd = d; rinv = inv_d;
                    off = top_of(); rec = NO_INST; iter = 0;
                    sp = 0; base = NO_BASE;
                    if ((Lane::ON ? view.units() : one_units) != 0) {
                        if (off >= (Lane::ON ? view.scene(one).n_nodes : one.n_nodes)) trip();
                        else {
                            const uint4* q = nodes() + 2ull * off;
                            const uint4 x = __ldg(q), y = __ldg(q + 1);
                            float tn;
                            if (box_hit(o, inv_d, x, y, t, tn)) {
                                count = min(y.w, IDLE - 1u);
                                at = count == 0 ? x.w + off : x.w;
                            }
                        }
                    }
                }
            }
            continue;
        }
        if (busy == 0) break;
        // The lanes at an interior node, at a unit, at triangles (the last two counted only when they could be more).
        const int n_inner = __popc(__ballot_sync(ALL, count == 0)), n_leaf = n_busy - n_inner;
        unsigned units = 0;
        if (n_inner < n_leaf) units = __ballot_sync(ALL, count - 1u < IDLE - 1u && rec == NO_INST);
        const int n_unit = __popc(units), n_tri = n_leaf - n_unit;
        if (n_inner >= n_leaf || n_inner >= max(n_unit, n_tri)) {
#pragma unroll
            for (int step = 0; step < STREAM_STEPS; ++step) {
                if (count == 0) {
                    if (iter++ >= WALK_GUARD || at >= last_node()) trip();
                    else {
                        const uint4* q = nodes() + 2ull * at;
                        const uint4 l0 = __ldg(q), l1 = __ldg(q + 1), r0 = __ldg(q + 2), r1 = __ldg(q + 3);
                        float tl, tr;
                        const bool hl = box_hit(ro, rinv, l0, l1, t, tl), hr = box_hit(ro, rinv, r0, r1, t, tr);
                        if (hl || hr) {
                            const bool swap = hr && (!hl || tr < tl);
                            const uint32_t link = swap ? r0.w : l0.w;
                            count = min(swap ? r1.w : l1.w, IDLE - 1u);
                            if (hl && hr && sp < 64) stack[sp++] = swap ? at : at + 1u;
                            at = count == 0 ? link + off : link;
                        } else {
                            pop();
                        }
                    }
                }
            }
        } else if (n_unit >= n_tri) {
            if (units >> lane & 1u) {
                uint32_t b, tables_end;
                const uint4* tables;
                if constexpr (Lane::ON) {
                    tables = view.scene(one).tables;
                    b = view.instances() + at * 10u;
                    tables_end = end32(view.scene(one).n_table_vec4);
                } else {
                    tables = one.tables;
                    b = one_instances + at * 10u;
                    tables_end = one_tables;
                }
                if (iter++ >= WALK_GUARD || tables_end < 10u || b > tables_end - 10u) trip();
                else {
                    const uint4* u = tables + b;
                    const float4* uf = reinterpret_cast<const float4*>(u);
                    const float4 n1 = __ldg(uf + 4);
                    const uint32_t ubits = bu(n1.w);
                    if (mode != TRACE_SHADOW || (ubits & UNIT_SHADOW) != 0) {
                        const float4 n0 = __ldg(uf + 3), n2 = __ldg(uf + 5);
                        rec = at;
                        ro = o - V3{__ldg(&uf[0].w), __ldg(&uf[1].w), __ldg(&uf[2].w)};
                        first = __ldg(&u[6].x);
                        if ((ubits & UNIT_SHIFTED) == 0) {
                            ro = proc_dir(n0, n1, n2, ro);
                            rd = proc_dir(n0, n1, n2, d);
                            rinv = safe_inv(rd);
                        }
                        off = bu(n0.w);
                        base = sp;
                        if (off > last_node()) trip();
                        else {
                            const uint32_t* q = reinterpret_cast<const uint32_t*>(nodes() + 2ull * off);
                            at = __ldg(q + 3);
                            count = min(__ldg(q + 7), IDLE - 1u);
                            if (count == 0) at += off;
                        }
                    } else {
                        pop();
                    }
                }
            }
        } else if (count - 1u < IDLE - 1u && rec != NO_INST) {
            const DScene& S = view.scene(one);
            const uint32_t tris_end = Lane::ON ? end32(S.n_tris) : one_tris;
            bool ended = iter++ >= WALK_GUARD;
            if (ended) trip();
            for (uint32_t k = 0; !ended && k < count; ++k) {
                const uint32_t ti = first + at + k;
                if (ti >= tris_end) { trip(); ended = true; break; }
                const float3 x = intersect_tri(S, ro, rd, ti, t);
                if (x.x < t) {
                    t = x.x;
                    if (hit(ray, x, ti, rec)) { count = IDLE; ended = true; break; }
                }
            }
            if (!ended) pop();
        }
        __syncwarp();
    }
    if (ray != NO_RAY) done(ray);
}

}  // namespace trt
