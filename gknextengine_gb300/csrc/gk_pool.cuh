// gk_pool.cuh — pools of paths and the warp-level ray scheduler of the path-tracing kernels (sm_103a).
//
// Each warp of a persistent kernel owns a pool of paths in device memory and alternates two phases
// over it: trace_queue traces the rays of the pool (a lane whose ray is finished takes the next one),
// then the kernel's own logic runs every path whose ray is answered up to its next ray. Path data is
// read and written past L1 (__ldcg / __stcg): a pool is larger than L1, which serves the nodes.
#pragma once
#include "gk_trace.cuh"

namespace gk {

constexpr int kPoolThreads = 128;
constexpr int kPoolWarps = kPoolThreads / 32;

// A path's first three fields of 16 bytes, the same in every kernel: origin and tmax; direction and
// the kind of ray; and the answer (instance, primitive, triangle; instance 0xFFFFFFFF on a miss).
enum PoolField { PF_RAYO = 0, PF_RAYD, PF_HIT, PF_FIRST_OWN };
enum RayKind : uint32_t { kRayCamera = 0, kRayBounce = 1, kRayAny = 2 };

// Paths per warp, at most: a larger pool fills the shading phase's warps with paths of one kind and
// refills lanes for longer. 64 / 128 / 192 / 256 paths: 1080p bricks 3.94 / 3.20 / 3.14 / 3.05 ms,
// 4K city - / 58.4 / 55.1 / 53.3, textured - / 9.7 / 8.6 / 8.1; 480 paths (their state outgrows L2)
// 3.15 / 52.6 / 8.9.
constexpr uint32_t kPoolMax = 256;
// The traversal's schedule, in lanes: node tests run while at least kNodeLanes lanes have one, then
// instance transitions (kTransLanes waiting) or triangle leaves (kLeafLanes), and finished rays make
// room for new ones kRefillLanes at a time. kNodeLanes 8 / 12 / 16: 4K city 56.7 / 55.1 / 57;
// kTransLanes 4 / 8 / 12: 57.2 / 52.6 / 54.9; kLeafLanes 10 / 14: 52.6 / 55.2; kRefillLanes
// 4 / 6 / 8: 48.7 / 48.0 / 47.9 (1080p bricks 2.85 / 2.82 / 2.79, textured 6.38 / 6.30 / 6.23).
constexpr int kNodeLanes = 12, kTransLanes = 8, kLeafLanes = 10, kRefillLanes = 8;

// kOne: pools of one warp's worth of paths, which trace all their rays to the end before they shade again.
// Latency is all there is to the small frames that use them: their fields go through L1 (a few pools per
// SM; larger pools would drive out the nodes), there is no stash, and work runs for the fewer lanes the
// fewer are left. (Frames of bricks with fixed thresholds, then shares: 300 x 200 at 1 sample 324 -> 288 us,
// at 8 samples 1642 -> 1470.)
template <bool kOne>
__device__ __forceinline__ float4 pool_get(const float4* p) { return kOne ? *p : __ldcg(p); }
template <bool kOne>
__device__ __forceinline__ void pool_put(float4* p, float4 v) {
    if (kOne) *p = v;
    else __stcg(p, v);
}

// The paths of a warp's pool whose rays are finished, in three lists by the kind of ray (camera,
// bounce, any-hit): the shading phase takes full warps of one kind, so that its sections run for
// all lanes or not at all, and mixed ones only when no kind has a warp's worth.
typedef uint8_t PathId;
static_assert(kPoolMax <= 256, "PathId");
struct DoneLists {
    PathId* l;         // 3 x np entries
    uint32_t np;
    int n[3];          // warp-uniform
    __device__ int total() const { return n[0] + n[1] + n[2]; }
    __device__ int largest() const { return max(n[0], max(n[1], n[2])); }
    // Every lane of the warp calls it.
    __device__ void add(bool mine, uint32_t kind, uint32_t slot) {
        const unsigned below = (1u << (threadIdx.x & 31u)) - 1u;
#pragma unroll
        for (uint32_t q = 0; q < 3u; ++q) {
            const unsigned m = __ballot_sync(0xFFFFFFFFu, mine && kind == q);
            if (mine && kind == q) l[q * np + (uint32_t)(n[q] + __popc(m & below))] = (PathId)slot;
            n[q] += __popc(m);
        }
    }
    // Entry k of the `take` first entries of each list, in the order of the kinds.
    __device__ uint32_t at(int k, const int (&take)[3]) const {
        uint32_t base = 0;
        if (k >= take[0]) {
            k -= take[0];
            base = np;
            if (k >= take[1]) { k -= take[1]; base = 2u * np; }
        }
        return l[base + (uint32_t)k];
    }
    // Drops the `take` first entries of each list (what stays is less than a warp's worth, or all).
    __device__ void drop(const int (&take)[3]) {
        __syncwarp();
        const int lane = threadIdx.x & 31;
#pragma unroll
        for (int q = 0; q < 3; ++q) {
            const int left = n[q] - take[q];
            if (take[q] > 0 && left > 0) {
                PathId* p = l + (uint32_t)q * np;
                PathId v = 0;
                if (lane < left) v = p[take[q] + lane];
                __syncwarp();
                if (lane < left) p[lane] = v;
            }
            n[q] = left;
        }
        __syncwarp();
    }
};

// A list of paths, grown at its end by any of the warp's lanes.
struct PathList {
    PathId* l;
    int n;             // warp-uniform
    __device__ void add(bool mine, uint32_t slot) {   // every lane of the warp calls it
        const unsigned m = __ballot_sync(0xFFFFFFFFu, mine);
        if (mine) l[n + __popc(m & ((1u << (threadIdx.x & 31u)) - 1u))] = (PathId)slot;
        n += __popc(m);
    }
};

// The rays that a warp's lanes are in the middle of, kept over the shading phase: 8 float4 fields of
// 32 lanes each in device memory (the world ray and the stack stay in shared memory).
constexpr int kStashFields = 8;
// Device memory of a warp, in float4: its pool of np paths, and the stash that pools of one warp's worth
// do without.
__host__ __device__ constexpr uint32_t warp_pool_size(uint32_t fields, uint32_t np, bool one) {
    return fields * np + (one ? 0u : kStashFields * 32u);
}
__device__ __forceinline__ void stash_save(float4* s, const Trav& T, int st, uint32_t slot) {
    const unsigned flags = (unsigned)st | (T.hit ? 4u : 0u) | (T.best_exact ? 8u : 0u) | (T.inblas ? 16u : 0u) |
                           ((unsigned)T.mode << 5) | (slot << 8);
    __stcg(s, make_float4(T.sl.inv.x, T.sl.inv.y, T.sl.inv.z, __uint_as_float(flags)));
    __stcg(s + 32, make_float4(T.sl.nn.x, T.sl.nn.y, T.sl.nn.z, T.tmax));
    __stcg(s + 64, make_float4(T.sl.nf.x, T.sl.nf.y, T.sl.nf.z, T.tcull));
    __stcg(s + 96, make_float4(T.o.x, T.o.y, T.o.z, T.best_lo));
    __stcg(s + 128, make_float4(T.d.x, T.d.y, T.d.z, T.best_hi));
    __stcg(s + 160, make_float4(__uint_as_float(T.inst), __uint_as_float(T.prim), __uint_as_float(T.tri),
                                __uint_as_float(T.cur)));
    __stcg(s + 192, make_float4(__int_as_float(T.ref), __int_as_float(T.sp), __int_as_float(T.iter), 0.0f));
    __stcg(s + 224, make_float4(__int_as_float(__double2loint(T.best_td)), __int_as_float(__double2hiint(T.best_td)),
                                0.0f, 0.0f));
}
__device__ __forceinline__ void stash_load(const float4* s, Trav& T, int& st, uint32_t& slot) {
    const float4 a = __ldcg(s), b = __ldcg(s + 32), c = __ldcg(s + 64), d = __ldcg(s + 96), e = __ldcg(s + 128),
                 f = __ldcg(s + 160), g = __ldcg(s + 192), h = __ldcg(s + 224);
    const unsigned flags = __float_as_uint(a.w);
    st = (int)(flags & 3u);
    T.hit = (flags & 4u) != 0u; T.best_exact = (flags & 8u) != 0u; T.inblas = (flags & 16u) != 0u;
    T.mode = (int)((flags >> 5) & 1u);
    slot = flags >> 8;
    T.sl.inv = F3(a.x, a.y, a.z); T.sl.nn = F3(b.x, b.y, b.z); T.sl.nf = F3(c.x, c.y, c.z);
    T.tmax = b.w; T.tcull = c.w; T.best_lo = d.w; T.best_hi = e.w;
    T.o = F3(d.x, d.y, d.z); T.d = F3(e.x, e.y, e.z);
    T.inst = __float_as_uint(f.x); T.prim = __float_as_uint(f.y); T.tri = __float_as_uint(f.z);
    T.cur = __float_as_uint(f.w);
    T.ref = __float_as_int(g.x); T.sp = __float_as_int(g.y); T.iter = __float_as_int(g.z);
    T.best_td = __hiloint2double(__float_as_int(h.y), __float_as_int(h.x));
}

constexpr uint32_t kNoSlot = 0x3FFu;     // pools hold fewer paths
// No ray in flight.
__device__ __forceinline__ void stash_empty(float4* s, const SceneView& S) {
    Trav T;
    trav_init(T, S, F3(0.0f, 0.0f, 0.0f), F3(1.0f, 0.0f, 0.0f), 1.0f, kClosest);
    stash_save(s, T, kStDone, kNoSlot);
}

// Traces rays of the queue until it is empty and the shading phase has a warp's worth of finished
// rays (or no ray is left). Every step runs one kind of work for all the lanes that need it: node tests while
// at least kNodeLanes lanes have one, else instance transitions or triangle leaves, whichever
// enough lanes wait for; lanes without a ray take one from the queue. The rays the lanes are in the
// middle of at the end stay in the stash, so that a warp never waits for its longest ray.
template <bool kOne = false>
__device__ __forceinline__ void trace_queue(const SceneView& S, PathList& queue, DoneLists& done, float4* pool, uint32_t np,
                                            float4* stash, float* wray, uint32_t* stk, int cap, Counters& cn) {
    int kN = kNodeLanes, kT = kTransLanes, kL = kLeafLanes;
    Trav T;
    int st;
    uint32_t slot;
    if (kOne) {   // every ray of the last time was finished
        st = kStDone;
        slot = kNoSlot;
    } else {
        stash_load(stash, T, st, slot);
    }
    uint32_t kind = slot >> 10;
    slot &= kNoSlot;
    bool have = slot != kNoSlot;
    int waiting = 0;                // entries taken from the queue's front
    // finished rays that the shading phase takes mixed (94 hold a warp's worth of one of the three
    // kinds); a pool of one warp's worth is traced to its end
    const int enough = !kOne && np >= 64u ? min(94, (int)np - 32) : (int)np + 1;
    bool alone = false;             // node tests for fewer lanes than kNodeLanes, for want of other work
    for (;;) {
        unsigned mn = __ballot_sync(0xFFFFFFFFu, st == kStNode);
        // node tests
        if (__popc(mn) >= kN || alone) {
            alone = false;
            do {
                if (st == kStNode) st = trav_node(T, S, stk, kPoolThreads, cn, cap);
                mn = __ballot_sync(0xFFFFFFFFu, st == kStNode);
            } while (__popc(mn) >= kN);
        }
        const unsigned md = __ballot_sync(0xFFFFFFFFu, st == kStDone);
        const bool more = waiting < queue.n;
        if (kOne && !more) {   // no ray will join: the thresholds are shares of the rays left
            const int n = 32 - __popc(md);
            kN = max(1, n >> 1);
            kT = max(1, (3 * n) >> 3);
            kL = max(1, (5 * n) >> 4);
        }
        const bool refill = more && (__popc(md) >= kRefillLanes || md == 0xFFFFFFFFu);
        if (refill || !more) {
            // finished rays to their paths
            const bool fin = have && st == kStDone;
            if (__any_sync(0xFFFFFFFFu, fin)) {
                if (fin) {
                    pool_put<kOne>(pool + slot + PF_HIT * np,
                                   make_float4(__uint_as_float(T.hit ? T.inst : 0xFFFFFFFFu), __uint_as_float(T.prim),
                                               __uint_as_float(T.tri), 0.0f));
                    have = false;
                }
                done.add(fin, kind, slot);
            }
            if (refill) {   // the next rays of the queue to the free lanes
                const int k = waiting + __popc(md & ((1u << (threadIdx.x & 31u)) - 1u));
                if (st == kStDone && k < queue.n) {
                    slot = queue.l[k];
                    const float4 o = pool_get<kOne>(pool + slot + PF_RAYO * np), d = pool_get<kOne>(pool + slot + PF_RAYD * np);
                    kind = __float_as_uint(d.w);
                    trav_init(T, S, F3(o.x, o.y, o.z), F3(d.x, d.y, d.z), o.w, kind == kRayAny ? kAny : kClosest);
                    wray[0] = o.x; wray[kPoolThreads] = o.y; wray[2 * kPoolThreads] = o.z;
                    wray[3 * kPoolThreads] = d.x; wray[4 * kPoolThreads] = d.y; wray[5 * kPoolThreads] = d.z;
                    st = T.done ? kStDone : kStNode;
                    have = true;
                }
                waiting = min(queue.n, waiting + __popc(md));
                continue;
            }
            // no ray left, or back to the shading phase if it has work
            if (md == 0xFFFFFFFFu || (!kOne && (done.largest() >= 32 || done.total() >= enough))) break;
        }
        const unsigned mx = __ballot_sync(0xFFFFFFFFu, st == kStTrans), ml = __ballot_sync(0xFFFFFFFFu, st == kStLeaf);
        if (__popc(mx) >= kT || (mx != 0u && mn == 0u && __popc(mx) >= __popc(ml))) {
            if (st == kStTrans) {
                T.wo = F3(wray[0], wray[kPoolThreads], wray[2 * kPoolThreads]);
                T.wd = F3(wray[3 * kPoolThreads], wray[4 * kPoolThreads], wray[5 * kPoolThreads]);
                st = trav_trans(T, S, stk, kPoolThreads, cap);
            }
        } else if (__popc(ml) >= kL || (ml != 0u && mn == 0u)) {
            if (st == kStLeaf) {
                T.wo = F3(wray[0], wray[kPoolThreads], wray[2 * kPoolThreads]);
                T.wd = F3(wray[3 * kPoolThreads], wray[4 * kPoolThreads], wray[5 * kPoolThreads]);
                st = trav_tris(T, S, stk, kPoolThreads, cn);
            }
        } else {
            alone = true;   // mn != 0 here: mx and ml below their thresholds
        }
    }
    queue.n = 0;
    if (!kOne) stash_save(stash, T, have ? st : kStDone, have ? (slot | (kind << 10)) : kNoSlot);
    __syncwarp();
}

// Shared memory words per thread beside the stack: the world ray in flight.
constexpr int kPoolRayWords = 6;
// Bytes of a block's path lists: three done lists, the queue and the spare list per warp.
constexpr size_t pool_list_bytes(uint32_t np) { return (size_t)5 * np * kPoolWarps * sizeof(PathId); }

}  // namespace gk
