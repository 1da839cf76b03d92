// gk_query.cuh — the warp-level loop of the ray-query kernels (sm_103a).
//
// A persistent warp answers rays of an array, every `warps`-th run of `per` rays of it (`per` lanes
// at work). A lane whose ray is finished takes the warp's next one, every step runs one kind of
// traversal work for all the lanes that need it (gk_pool.cuh's schedule), and the answers are
// completed and written 32 at a time from a ring in shared memory: a ray's hit record is written
// only after the ray was read for the last time, so that rays and hits may share one buffer.
#pragma once
#include "../../include/gkrt.h"
#include "gk_pool.cuh"

namespace gk {

constexpr int kQueryThreads = 128;
constexpr int kQueryWarps = kQueryThreads / 32;
constexpr int kQueryRefillLanes = 4;   // finished rays make room for new ones so many at a time
constexpr int kQueryRing = 64;      // finished rays per warp: fewer than 32 kept, up to 32 more per step
// Shared memory of a block: stacks and world rays per thread, a ring of 16-byte entries per warp.
constexpr size_t query_smem(int stack_words) {
    return (size_t)(stack_words + kPoolRayWords) * kQueryThreads * 4u + (size_t)kQueryWarps * kQueryRing * 16u;
}

// Rays per warp run and blocks for `n` rays: few rays are spread over as many warps as the device
// holds (a warp's rays wait for one another), many fill every lane.
__host__ inline void query_grid(uint32_t n, int num_sms, int blocks_per_sm, uint32_t& blocks, uint32_t& per) {
    const uint32_t most = (uint32_t)num_sms * (uint32_t)(blocks_per_sm < 1 ? 1 : blocks_per_sm);
    const uint64_t warps = (uint64_t)most * kQueryWarps;
    per = n < 32u * warps ? (uint32_t)((n + warps - 1) / warps) : 32u;
    if (per < 1u) per = 1u;
    const uint64_t need = ((uint64_t)n + (uint64_t)per * kQueryWarps - 1) / ((uint64_t)per * kQueryWarps);
    blocks = (uint32_t)(need < most ? need : most);
}

// Ray i: two 16-byte loads where the array allows them (wide), else eight words, as any 4-byte
// aligned array was always taken.
__device__ __forceinline__ void query_load(const GkrtRay* rays, uint32_t i, bool wide, float4& o, float4& d) {
    if (wide) {
        const float4* p = reinterpret_cast<const float4*>(rays + i);
        o = p[0];
        d = p[1];
    } else {
        const GkrtRay& r = rays[i];
        o = make_float4(r.origin[0], r.origin[1], r.origin[2], r.tmin);
        d = make_float4(r.dir[0], r.dir[1], r.dir[2], r.tmax);
    }
}

// The arrays of a ray query as a source of query_run.
struct QueryRays {
    const SceneView& S;
    const GkrtRay* rays;
    GkrtHit* hits;
    bool any, wide;
    // Ray k: origin and tmin, direction and tmax; true for an any-hit ray.
    __device__ bool load(uint32_t k, float4& o, float4& d) const {
        query_load(rays, k, wide, o, d);
        return any;
    }
    // The answer e = (ray, instance or 0xFFFFFFFF, primitive, triangle).
    __device__ void write(const uint4& e, Counters& cn) const {
        float t = -1.0f, b1 = 0.0f, b2 = 0.0f;
        uint32_t prim = 0xFFFFFFFFu;
        if (e.y != 0xFFFFFFFFu) {
            ++cn.hits;
            float4 o, d;
            query_load(rays, e.x, wide, o, d);
            const HitShade s = hit_shade(S, F3(o.x, o.y, o.z), F3(d.x, d.y, d.z), e.y, e.w);
            t = s.t;
            prim = e.z;
            if (!any) { b1 = s.b1; b2 = s.b2; }
        }
        if (wide) {
            float4* h = reinterpret_cast<float4*>(hits + e.x);
            h[0] = make_float4(t, b1, b2, __uint_as_float(e.y));
            h[1] = make_float4(__uint_as_float(prim), 0.0f, 0.0f, 0.0f);
        } else {
            GkrtHit& h = hits[e.x];
            h.t = t; h.b1 = b1; h.b2 = b2; h.inst = e.y; h.prim = prim;
            h.pad[0] = h.pad[1] = h.pad[2] = 0u;
        }
    }
};

// smem: query_smem(cap) bytes of the block's dynamic shared memory, 16-byte aligned. src.load is called
// once per ray, src.write by up to 32 lanes together, for rays that load was called for before.
template <class Source>
__device__ __forceinline__ void query_run(const SceneView& S, const Source& src, uint32_t n, uint32_t per, int cap,
                                          uint32_t* smem, Counters& cn) {
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    uint4* ring = reinterpret_cast<uint4*>(smem) + warp * kQueryRing;
    uint32_t* stk = smem + kQueryWarps * kQueryRing * 4 + tid;
    float* wray = reinterpret_cast<float*>(smem + kQueryWarps * kQueryRing * 4 + cap * kQueryThreads) + tid;
    const uint64_t warps = (uint64_t)gridDim.x * kQueryWarps, me = (uint64_t)blockIdx.x * kQueryWarps + warp;
    // ray s of this warp is ray ((s / per) warps + me) per + s mod per of the array
    uint64_t run = me * per;            // first ray of the current run
    uint32_t off = 0;                   // rays of it that were taken
    int ringn = 0, st = kStDone;
    bool have = false;
    uint32_t ray = 0;
    Trav T;
    const unsigned below = (1u << lane) - 1u;
    for (;;) {
        unsigned mn = __ballot_sync(0xFFFFFFFFu, st == kStNode);
        const int thr = per < 32u ? 1 : kNodeLanes;
        if (__popc(mn) >= thr) {
            do {
                if (st == kStNode) st = trav_node<true>(T, S, stk, kQueryThreads, cn, cap);
                mn = __ballot_sync(0xFFFFFFFFu, st == kStNode);
            } while (__popc(mn) >= thr);
        }
        const unsigned md = __ballot_sync(0xFFFFFFFFu, st == kStDone);
        if (__popc(md) >= kQueryRefillLanes && (run < n || md == 0xFFFFFFFFu || __any_sync(0xFFFFFFFFu, have && st == kStDone))) {
            // finished rays to the ring, complete entries written, the next rays to the free lanes
            const bool fin = have && st == kStDone;
            const unsigned mf = __ballot_sync(0xFFFFFFFFu, fin);
            if (fin) {
                ring[ringn + __popc(mf & below)] =
                    make_uint4(ray, T.hit ? T.inst : 0xFFFFFFFFu, T.prim, T.tri);
                have = false;
            }
            ringn += __popc(mf);
            __syncwarp();
            if (ringn >= 32) {
                src.write(ring[lane], cn);
                __syncwarp();
                const int left = ringn - 32;
                uint4 e = make_uint4(0u, 0u, 0u, 0u);
                if (lane < left) e = ring[32 + lane];
                __syncwarp();
                if (lane < left) ring[lane] = e;
                ringn = left;
                __syncwarp();
            }
            if (run < n) {
                const uint32_t k = off + (uint32_t)__popc(md & below);
                const uint64_t r = run + k;
                if (st == kStDone && k < per && r < n) {
                    ray = (uint32_t)r;
                    float4 o, d;
                    const bool any = src.load(ray, o, d);
                    ++cn.rays;
                    trav_init(T, S, F3(o.x, o.y, o.z), F3(d.x, d.y, d.z), d.w, any ? kAny : kClosest, o.w);
                    wray[0] = o.x; wray[kQueryThreads] = o.y; wray[2 * kQueryThreads] = o.z;
                    wray[3 * kQueryThreads] = d.x; wray[4 * kQueryThreads] = d.y; wray[5 * kQueryThreads] = d.z;
                    st = T.done ? kStDone : kStNode;
                    have = true;
                }
                off += (uint32_t)__popc(md);
                if (off >= per) {
                    off = 0;
                    run += warps * per;
                }
            } else if (__ballot_sync(0xFFFFFFFFu, have) == 0u) {
                break;
            }
            continue;
        }
        const unsigned mx = __ballot_sync(0xFFFFFFFFu, st == kStTrans), ml = __ballot_sync(0xFFFFFFFFu, st == kStLeaf);
        if (__popc(mx) >= kTransLanes || (mx != 0u && mn == 0u && __popc(mx) >= __popc(ml))) {
            if (st == kStTrans) {
                T.wo = F3(wray[0], wray[kQueryThreads], wray[2 * kQueryThreads]);
                T.wd = F3(wray[3 * kQueryThreads], wray[4 * kQueryThreads], wray[5 * kQueryThreads]);
                st = trav_trans(T, S, stk, kQueryThreads, cap);
            }
        } else if (__popc(ml) >= kLeafLanes || (ml != 0u && mn == 0u)) {
            if (st == kStLeaf) {
                T.wo = F3(wray[0], wray[kQueryThreads], wray[2 * kQueryThreads]);
                T.wd = F3(wray[3 * kQueryThreads], wray[4 * kQueryThreads], wray[5 * kQueryThreads]);
                st = trav_tris<true>(T, S, stk, kQueryThreads, cn);
            }
        } else if (st == kStNode) {     // some lane has a node: the other kinds wait below their thresholds
            st = trav_node<true>(T, S, stk, kQueryThreads, cn, cap);
        }
    }
    if (lane < ringn) src.write(ring[lane], cn);
    __syncwarp();
}

__device__ __forceinline__ void query_rays(const SceneView& S, const GkrtRay* rays, GkrtHit* hits, uint32_t n, uint32_t mode,
                                           uint32_t per, int cap, uint32_t* smem, Counters& cn) {
    const bool wide = ((reinterpret_cast<uintptr_t>(rays) | reinterpret_cast<uintptr_t>(hits)) & 15u) == 0u;
    const QueryRays src{S, rays, hits, mode == GKRT_TRACE_ANY, wide};
    query_run(S, src, n, per, cap, smem, cn);
}

}  // namespace gk
