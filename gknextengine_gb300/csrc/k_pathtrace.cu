// k_pathtrace.cu — the "rt pass" (Core.PathTracing) and ray-query kernels for sm_103a.
//
// The rt pass is one persistent kernel: every path runs the per-pixel logic of
// FPathTracingRendererV2 (assets/shaders/common/Shading.slang:1084-1241, with the traced
// camera ray of FHardwarePrimaryRayCaster, :283-334) as a state machine that stops
// whenever it needs a ray traced. Each warp owns a pool of paths in device memory (a few per
// lane; the pools of a large frame are larger than L2) and alternates two phases over it: all rays of the pool are traced, a lane
// whose ray is finished taking the next one, then every path runs its state machine to its next
// ray, 32 paths of one kind at a time, and pixels from a global counter (8 x 4 pixel tiles) take
// the places of paths that ended. A warp thus waits for its longest ray once per pool instead of
// once per 32 rays, and neither phase carries the other's state in registers. Each path keeps
// its own RNG stream, so results do not depend on the schedule.
#include <algorithm>

#include "gk_query.cuh"
#include "gk_shade.cuh"
#include "gkrt_internal.h"

namespace gk {

constexpr int kPtThreads = kPoolThreads;
constexpr int kPtWarps = kPoolWarps;
// Resident blocks per SM, at most (what the pools are sized for): the traversal phase fits 128 registers, the
// shading phase spills below.
// Trace pass with 3 / 4 / 5 blocks (ms): 1080p bricks 3.12 / 2.84 / 3.03, Cornell 256 x 256
// 0.160 / 0.134 / 0.150, 720p on the probe grid 1.31 / 1.16 / 1.14, 4K city 52.3 / 48.7 / 48.4, textured
// 1277 x 713 at 8 samples 6.8 / 6.6 / 7.7.
constexpr int kPtBlocks = 4;
// Pools of one warp's worth (kOne) serve frames of up to kPtOneWarps warps' worth of pixels per SM, with
// three blocks per SM, whose registers hold a path almost without spills (32 to 56 bytes), or two, which have
// none, where those have a lane for every pixel. Whole frames of bricks with 2 / 3 / 4 /
// 5 blocks, us: 100 x 70 pixels 215 / 220 / 231 / 272, 300 x 200 250 / 269 / 288 / 330, 400 x 300 358 / 305 /
// 333 / 406; Cornell 256 x 256 158 / 131 / 156 / 176. One-warp pools / larger ones, us, at 640 x 400 (53
// warps' worth per SM): bricks 554 / 560, Cornell 325 / 312, textured 556 / 482, field of bricks on the probe
// grid 515 / 533, city 1545 / 1548; at 700 x 400 (58): 602 / 588, 339 / 325, 586 / 501, 557 / 549, 1664 / 1648.
constexpr uint32_t kPtOneWarps = 56;
constexpr float kCosCone = 0.999990482f;   // cos(0.25 deg), Shading.slang:897

// Warp-aggregated flush: one atomic per counter per warp. Slots 0-5 are per pass
// (rays, FP64 fallbacks, exact re-traces, node visits, triangle tests, hit fetches); slot 6
// counts rays since the context was created.
__device__ __forceinline__ void flush_counters(const Counters& c, unsigned long long* out) {
    unsigned long long v[6] = {c.rays, c.fallbacks, c.retraces, c.nodes, c.tris, c.hits};
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
#pragma unroll
        for (int k = 0; k < 6; ++k) v[k] += __shfl_down_sync(0xFFFFFFFFu, v[k], o);
    if ((threadIdx.x & 31) == 0) {
#pragma unroll
        for (int k = 0; k < 6; ++k)
            if (v[k]) atomicAdd(&out[k], v[k]);
        if (v[0]) atomicAdd(&out[6], v[0]);
    }
}

enum Stage : uint32_t {
    ST_PRIMARY = 0, ST_FIRST = 1, ST_BOUNCE = 2, ST_SUN = 3, ST_DIRECT = 4,
    ST_NEE_FIRST = 5, ST_NEE_BOUNCE = 6   // emissive-triangle shadow ray before the first / a later bounce
};

// A path in its warp's pool: fields of 16 bytes, field f of the pool's paths contiguous, so that 32
// paths are read and written as whole lines. The ray and its hit, the RNG state, the throughput
// and the state word travel every time; the current vertex and direction only over any-hit rays
// (a bounce ray's vertex is its hit, its direction its own); the primary vertex, the loop bounds,
// the two accumulators, the pending emissive-NEE sample and (textured scenes) the primary albedo
// are read where the logic needs them.
enum Field {
    PF_SEED = PF_FIRST_OWN, PF_RC, PF_STATE, PF_VP, PF_VN, PF_DIR, PF_PP, PF_PN, PF_FC, PF_FR, PF_NEE,
    PF_ALB, PF_COUNT
};
static_assert(PF_COUNT == kPathPoolFields, "pool size");

// The ray a path stops at, and its answer.
struct PathRay {
    f3 wo, wd;
    float tmax;
    bool any;                    // any-hit (shadow) or closest-hit ray
    bool hit;
    uint32_t inst, prim, tri;
};

struct Lane {
    int pix;          // pixel index
    Rng seed;
    uint32_t stage;
    uint32_t i, b;    // sample and bounce indices
    bool chanceReflect, back, diel, hitReflect, hitMetal;
    bool neeLobe;     // the bounce in flight was sampled from the diffuse lobe of an emissive-NEE vertex
    f4 rc;            // throughput of the current sample (RayColor)
    Vtx vs;           // current path vertex
    f3 dir;           // current path direction
};

template <bool kOne>
struct Ctx {
    const ShadeScene& sc;
    const GkrtFrameConstants& fc;
    const PixelImages& im;
    int W, H, P;      // P: image row pitch in pixels
    float4* path;     // this path's field 0
    uint32_t np;      // paths per pool: the stride between fields
    Counters& cn;
    __device__ f4 get(int f) const {
        const float4 v = pool_get<kOne>(path + (uint32_t)f * np);
        return F4(v.x, v.y, v.z, v.w);
    }
    __device__ void put(int f, f4 v) const {
        pool_put<kOne>(path + (uint32_t)f * np, make_float4(v.x, v.y, v.z, v.w));
    }
    __device__ void put(int f, f3 v, uint32_t w) const { put(f, F4(v.x, v.y, v.z, __uint_as_float(w))); }
};

template <class Ctx>
__device__ __forceinline__ void emit(PathRay& R, const Ctx& c, f3 o, f3 d, bool any, float tmax = 1000.0f) {
    ++c.cn.rays;
    R.wo = o; R.wd = d; R.tmax = tmax; R.any = any;
}

// primaryAlbedo_ of the reference: the material's diffuse, times its diffuse texture (kTex)
template <bool kTex, class Ctx>
__device__ __forceinline__ f4 pv_albedo(const Ctx& c) {
    if (kTex) return c.get(PF_ALB);
    return load_mat(c.sc, __float_as_uint(c.get(PF_PP).w)).diffuse;
}

// Run the lane's state machine on the ray that just finished, up to the next ray
// (returns true) or the end of the pixel (returns false). Follows FPathTracingRendererV2:
// PrimaryHit (Shading.slang:1186-1223), Render (:1084-1184) with GetRayColor
// (:1003-1082) split at its trace, the sun test of the bounce loop (:1135-1144), early exit
// and probe termination (:1146-1154), and DirectIlluminate (:886-908).
//
// The logic is laid out as guarded sections in one fixed order; every lane passes each
// section at most once per call, so lanes in different states re-converge after each
// section and the expensive ones (the hit reconstruction after a trace, the sampling before the
// next) run once per warp for all the lanes that need them.
// kTex: textured materials and the textured sky compiled in (the scene has texture ids or the
// frame samples a sky texture).
template <bool kNee, bool kTex, class Ctx>
__device__ __forceinline__ bool advance(Lane& L, PathRay& T, const Ctx& c) {
    const GkrtFrameConstants& fc = c.fc;
    const f3 sunDir = F3(fc.sun_direction[0], fc.sun_direction[1], fc.sun_direction[2]);
    const uint32_t stage = L.stage;
    bool emitted = false, need_begin = false, need_pre = false, pre_first = false;
    bool need_end = false, need_after_sun = false, need_finish = false;
    bool need_probe = false, need_sun = false;
    float shadow = 0.0f;
    f3 sunO;   // where the sun ray starts

    // 0. the vertex a closest-hit ray met
    HitVtx hv;
    if (stage <= ST_BOUNCE && T.hit) {
        ++c.cn.hits;
        hv = hit_vertex(c.sc, T.wo, T.wd, T.inst, T.prim, T.tri);
    }

    // 1. the camera ray's hit: G-buffer outputs, motion, sample set-up
    if (stage == ST_PRIMARY) {
        const int pix = L.pix;
        const bool want_ids = (fc.flags & GKRT_FRAME_PRIMARY_IDS) != 0u;
        c.im.single_specular[pix] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        if (!T.hit) {
            const f4 s = kTex ? sky_dir(c.sc, fc, normalize3(T.wd)) : sky(fc);
            c.im.single_diffuse[pix] = make_float4(s.x, s.y, s.z, s.w);
            c.im.motion[pix] = make_float2(0.0f, 0.0f);
            c.im.albedo[pix] = make_float4(1.0f, 1.0f, 1.0f, 1.0f);
            c.im.normal[pix] = make_float4(0.0f, 1.0f, 0.0f, 1.0f);
            c.im.object_id[pix] = 65535u;
            c.im.prev_depth[pix] = 100000.0f;
            if (want_ids) { c.im.hit_inst[pix] = 0xFFFFFFFFu; c.im.hit_prim[pix] = 0xFFFFFFFFu; }
        } else {
            Vtx pv = hv;
            if (want_ids) { c.im.hit_inst[pix] = T.inst; c.im.hit_prim[pix] = T.prim; }
            const f4 P4 = F4(pv.P.x, pv.P.y, pv.P.z, 1.0f);
            const f4 clip = mat4v(fc.view_projection, P4);
            const f4 ch = mat4v(fc.view_projection_unjit, P4);
            const float cfx = div_(ch.x, ch.w) * 0.5f, cfy = div_(ch.y, ch.w) * 0.5f;
            float cp[12];
#pragma unroll
            for (int q = 0; q < 12; ++q) cp[q] = __ldg(&c.sc.inst_prev[24u * pv.inst + q]);
            const f3 prevP = xpoint(cp, pv.P);
            const f4 ph = mat4v(fc.prev_view_projection_unjit, F4(prevP.x, prevP.y, prevP.z, 1.0f));
            const float pfx = div_(ph.x, ph.w) * 0.5f, pfy = div_(ph.y, ph.w) * 0.5f;
            uint32_t mom = c.im.motion_moment[pix];
            if (len3(pv.P - prevP) > 0.02f) mom = fc.temporal_frames;
            else mom = mom > 0u ? mom - 1u : 0u;
            c.im.motion_moment[pix] = mom;
            const MatV pm = load_mat(c.sc, pv.mat);
            f4 palb = pm.diffuse;
            float prough = pm.fuzz;
            if (kTex) {   // FetchGBufferV2 (Shading.slang:82-112)
                const HitAttr ha = hit_attr(c.sc, hv.i0, hv.i1, hv.i2, hv.b1, hv.b2);
                const GBufTex g = fetch_gbuffer(c.sc, pm, ha, pv.N, pv.inst);
                palb = g.albedo;
                prough = g.rough;
                pv.N = g.n;
            }
            c.im.albedo[pix] = make_float4(palb.x, palb.y, palb.z, palb.w);
            c.im.normal[pix] = make_float4(pv.N.x, pv.N.y, pv.N.z, prough);
            c.im.object_id[pix] = __ldg(&c.sc.S.inst[pv.inst].instance_id);
            c.im.motion[pix] = make_float2((pfx - cfx) * (float)c.W, (pfy - cfy) * (float)c.H);
            c.im.prev_depth[pix] = div_(clip.z, clip.w);
            if (pm.model != GKRT_MAT_DIELECTRIC) pv.P = fma3(normalize3(T.wd), -0.03f, pv.P);
            if (pm.model == GKRT_MAT_DIFFUSE_LIGHT) {
                c.im.single_diffuse[pix] = make_float4(pm.diffuse.x, pm.diffuse.y, pm.diffuse.z, pm.diffuse.w);
            } else {
                const bool pdiel = pm.model == GKRT_MAT_DIELECTRIC;
                int samples = (int)fc.number_of_samples * (mom > 0u ? 4 : 1);
                if (samples < 1) samples = 1;
                if (samples > 0xFFFF) samples = 0xFFFF;
                uint32_t maxB = pdiel ? fc.max_number_of_bounces : fc.number_of_bounces;
                if (maxB > 0x7FFFu) maxB = 0x7FFFu;
                c.put(PF_PP, pv.P, pv.mat);
                c.put(PF_PN, pv.N, (uint32_t)samples | (maxB << 16) | (pdiel ? 0x80000000u : 0u));
                c.put(PF_FC, F4(0.0f, 0.0f, 0.0f, 0.0f));
                c.put(PF_FR, F4(0.0f, 0.0f, 0.0f, 0.0f));
                if (kTex) c.put(PF_ALB, palb);
                L.i = 0;
                need_begin = true;
            }
        }
    }

    // 2. GetRayColor after its trace (Shading.slang:1039-1081), then the bounce loop's sun test
    if (stage == ST_FIRST || stage == ST_BOUNCE) {
        bool term;
        if (T.hit) {
            L.vs = hv;
            const MatV hm = load_mat(c.sc, L.vs.mat);
            if (kNee && L.neeLobe && hm.model == GKRT_MAT_DIFFUSE_LIGHT) {
                // the emitter this diffuse bounce reached was sampled by the vertex's NEE
                L.rc = F4(0.0f, 0.0f, 0.0f, 0.0f);
                term = true;
            } else {
                f4 halb = hm.diffuse;
                if (kTex && hm.dtex >= 0) {   // the hit's diffuse texture (Shading.slang:1046-1050)
                    const HitAttr ha = hit_attr(c.sc, hv.i0, hv.i1, hv.i2, hv.b1, hv.b2);
                    halb = halb * tex_sample(c.sc.tex, hm.dtex, ha.u, ha.v);
                }
                if (hm.model == GKRT_MAT_DIFFUSE_LIGHT || !L.chanceReflect) L.rc = L.rc * halb;
                if (L.back && !L.diel) { L.rc = F4(0.5f, 0.5f, 0.5f, 0.0f); term = true; }
                else term = hm.model == GKRT_MAT_DIFFUSE_LIGHT;
            }
        } else {
            L.rc = L.rc * (kTex ? sky_dir(c.sc, fc, T.wd) : sky(fc));
            term = true;
        }
        const uint32_t loop = __float_as_uint(c.get(PF_PN).w);
        if (term) {
            need_end = true;
        } else if (stage == ST_FIRST) {
            const uint32_t maxB = (loop >> 16) & 0x7FFFu;
            const bool pdiel = (loop >> 31) != 0u;
            if (fc.fast_gather && !pdiel) {
                need_probe = true;
            } else {
                L.b = 1;
                if (L.b < maxB) need_pre = true;
                else need_end = true;
            }
        } else if (fc.has_sun && rnd1(L.seed) < 0.5f) {
            L.stage = ST_SUN;
            sunO = L.vs.P;
            need_sun = true;
        } else {
            need_after_sun = true;
        }
    }

    // 3. the sun test's answer
    if (stage == ST_SUN) {
        if (!T.hit) {
            L.rc = L.rc * F4(fc.sun_color[0], fc.sun_color[1], fc.sun_color[2], fc.sun_color[3]);
            need_end = true;
        } else {
            need_after_sun = true;
        }
    }

    // 4. early exit or last bounce: probe termination, else the next bounce
    if (need_after_sun) {
        const uint32_t loop = __float_as_uint(c.get(PF_PN).w);
        const uint32_t maxB = (loop >> 16) & 0x7FFFu;
        const bool pdiel = (loop >> 31) != 0u;
        const bool early = !pdiel && rnd1(L.seed) < 0.5f;
        if (L.b == maxB - 1u || early) {
            need_probe = true;
        } else {
            ++L.b;
            need_pre = true;
        }
    }
    if (need_probe) {
        L.rc = L.rc * probe_term(c.sc, L.vs.P, L.vs.N);
        need_end = true;
    }

    // 5. end of a sample (Shading.slang:1159-1176), then the next sample or DirectIlluminate
    if (need_end) {
        if (L.hitMetal) L.rc = L.rc * pv_albedo<kTex>(c);
        const int acc = L.hitReflect ? PF_FR : PF_FC;
        c.put(acc, c.get(acc) + L.rc);
        const uint32_t samples = __float_as_uint(c.get(PF_PN).w) & 0xFFFFu;
        if (++L.i < samples) {
            need_begin = true;
        } else if (fc.has_sun) {
            L.stage = ST_DIRECT;
            sunO = xyz(c.get(PF_PP));
            need_sun = true;
        } else {
            shadow = 0.0f;
            need_finish = true;
        }
    }

    // 6. DirectIlluminate's answer
    if (stage == ST_DIRECT) {
        shadow = T.hit ? 0.0f : 1.0f;
        need_finish = true;
    }

    // 6b. an emissive-NEE shadow ray's answer, then the bounce ray its vertex sampled
    if (kNee && (stage == ST_NEE_FIRST || stage == ST_NEE_BOUNCE)) {
        if (!T.hit) {
            const int acc = L.hitReflect ? PF_FR : PF_FC;
            c.put(acc, c.get(acc) + c.get(PF_NEE));
        }
        L.stage = stage == ST_NEE_FIRST ? ST_FIRST : ST_BOUNCE;
        emit(T, c, fma3(L.vs.N, 0.001f, L.vs.P), L.dir, false);
        emitted = true;
    }

    // 7. the pixel's outputs (Shading.slang:1175-1183)
    if (need_finish) {
        const f4 pn = c.get(PF_PN);
        const float dd = mx(dot3(sunDir, normalize3(xyz(pn))), 0.0f) * 0.318309886183790671538f;
        // the means over the samples (Shading.slang:1171-1172)
        const float fs = (float)(__float_as_uint(pn.w) & 0xFFFFu);
        f4 fcol = c.get(PF_FC), frefl = c.get(PF_FR);
        fcol = F4(div_(fcol.x, fs), div_(fcol.y, fs), div_(fcol.z, fs), div_(fcol.w, fs));
        frefl = F4(div_(frefl.x, fs), div_(frefl.y, fs), div_(frefl.z, fs), div_(frefl.w, fs));
        fcol = fcol + F4((fc.sun_color[0] * dd) * shadow, (fc.sun_color[1] * dd) * shadow,
                         (fc.sun_color[2] * dd) * shadow, (fc.sun_color[3] * dd) * shadow);
        c.im.single_diffuse[L.pix] = make_float4(fcol.x, fcol.y, fcol.z, fcol.w);
        c.im.single_specular[L.pix] = make_float4(frefl.x, frefl.y, frefl.z, frefl.w);
    }

    // 8. start of a sample (Shading.slang:1103-1117)
    if (need_begin) {
        const f4 eye = mat4v(fc.model_view_inverse, F4(0.0f, 0.0f, 0.0f, 1.0f));
        L.rc = F4(1.0f, 1.0f, 1.0f, 1.0f);
        const f4 pp = c.get(PF_PP);
        L.vs.P = xyz(pp);
        L.vs.N = xyz(c.get(PF_PN));
        L.vs.mat = __float_as_uint(pp.w);
        L.dir = normalize3(L.vs.P - xyz(eye));
        L.hitReflect = false;
        L.hitMetal = false;
        need_pre = true;
        pre_first = true;
    }

    // 9. GetRayColor up to its trace (Shading.slang:1007-1039), or a ray in the sun's cone: one sampled
    // direction about one axis for either (GGX, cosine hemisphere, cone)
    if (need_pre || need_sun) {
        MatV mat;
        bool diel = false, chanceReflect = false, chanceMetal = false, chanceGGX = false, back = false;
        float startPosOffset = 0.0f, niOverNt = 0.0f;
        f3 outward, axis = sunDir;
        if (need_pre) {
            mat = load_mat(c.sc, L.vs.mat);
            diel = mat.model == GKRT_MAT_DIELECTRIC;
            startPosOffset = diel ? 0.0f : 1.0f;
            const float dotValue = dot3(L.dir, L.vs.N);
            back = dotValue > 0.0f;
            outward = back ? -L.vs.N : L.vs.N;
            niOverNt = back ? mat.ri2 : div_(1.0f, mat.ri2);
            const float cosine = dotValue > 0.0f ? mat.ri * dotValue : -dotValue;
            const float reflectProb = schlick(cosine, mat.ri);
            chanceReflect = rnd1(L.seed) < reflectProb;
            chanceMetal = rnd1(L.seed) < mat.metal;
            chanceGGX = chanceReflect || chanceMetal;
            axis = chanceGGX ? reflect3(L.dir, outward) : outward;
        }
        f3 tb, bb;
        onb(axis, tb, bb);
        f3 wi, v;
        float alpha = 0.0f, r, z;
        if (chanceGGX) {
            const float roughness = sqrt_(mat.fuzz);
            alpha = roughness * roughness;
            v = F3(dot3(tb, axis), dot3(bb, axis), dot3(axis, axis));
            wi = normalize3(F3(v.x * alpha, v.y * alpha, v.z));
        }
        const f2 u = rnd2(L.seed);
        float sn, cs;
        sincos2pi(u.x, sn, cs);
        if (chanceGGX) {
            z = ggx_vndf_z(alpha, v, wi, u.y);
            r = sqrt_(sat(fmaf_(-z, z, 1.0f)));
        } else if (need_pre) {
            r = sqrt_(u.y);
            z = sqrt_(1.0f - u.y);
        } else {
            z = cone_z(kCosCone, u.y);
            r = sqrt_(fmaf_(-z, z, 1.0f));
        }
        v = F3(r * cs, r * sn, z);
        if (chanceGGX) {
            const f3 m = wi + v;
            v = normalize3(F3(m.x * alpha, m.y * alpha, m.z));
        }
        f3 tdir = to_world(v, tb, bb, axis);
        if (need_sun) {
            emit(T, c, sunO, tdir, true);
        } else {
            if (pre_first) { L.hitReflect = chanceGGX; L.hitMetal = chanceMetal; }
            if (diel && !chanceReflect) tdir = refract3(L.dir, outward, niOverNt);
            L.dir = tdir;
            L.chanceReflect = chanceReflect;
            L.back = back;
            L.diel = diel;
            L.neeLobe = kNee && !back && !diel && !chanceGGX;
            NeeSample ns;
            if (kNee && L.neeLobe && nee_sample(c.sc, L.seed, L.vs.P, L.vs.N, L.rc, ns)) {
                f4 contrib = ns.contrib;
                if (L.hitMetal) contrib = contrib * pv_albedo<kTex>(c);
                c.put(PF_NEE, contrib);
                L.stage = pre_first ? ST_NEE_FIRST : ST_NEE_BOUNCE;
                emit(T, c, ns.o, ns.dir, true, ns.tmax);
            } else {
                L.stage = pre_first ? ST_FIRST : ST_BOUNCE;
                emit(T, c, fma3(L.vs.N, 0.001f * startPosOffset, L.vs.P), tdir, false);
            }
        }
        emitted = true;
    }
    return emitted;
}

// Camera ray of FHardwarePrimaryRayCaster (Shading.slang:286-304) for pixel index pix.
template <class Ctx>
__device__ __forceinline__ void start_pixel(Lane& L, PathRay& T, const Ctx& c, int x, int y) {
    const GkrtFrameConstants& fc = c.fc;
    L.pix = y * c.P + x;
    L.seed.v[0] = (uint32_t)x; L.seed.v[1] = (uint32_t)y; L.seed.v[2] = fc.total_frames; L.seed.v[3] = 0u;
    float uvx = fmaf_(div_((float)x, (float)c.W), 2.0f, -1.0f);
    float uvy = fmaf_(div_((float)y, (float)c.H), 2.0f, -1.0f);
    if (fc.taa) {
        const uint32_t hi = fc.total_frames % 8u;
        uvx = uvx + div_(c_halton[2 * hi] - 0.5f, (float)c.W);
        uvy = uvy + div_(c_halton[2 * hi + 1] - 0.5f, (float)c.H);
    }
    const f2 disk = unit_disk(L.seed);
    const float ha = div_(fc.aperture, 2.0f);
    const float offx = ha * disk.x, offy = ha * disk.y;
    const f4 origin = mat4v(fc.model_view_inverse, F4(offx, offy, 0.0f, 1.0f));
    const f4 target = mat4v(fc.projection_inverse, F4(uvx, uvy, 1.0f, 1.0f));
    const f3 tn = normalize3(F3(fmaf_(target.x, fc.focus_distance, -offx), fmaf_(target.y, fc.focus_distance, -offy),
                                target.z * fc.focus_distance));
    const f4 direction = mat4v(fc.model_view_inverse, F4(tn.x, tn.y, tn.z, 0.0f));
    L.stage = ST_PRIMARY;
    emit(T, c, xyz(origin), xyz(direction), false);
}

// State word pair of a path: stage and flags, sample and bounce indices.
template <class Ctx>
__device__ __forceinline__ void store_path(const Ctx& c, const Lane& L, const PathRay& R) {
    c.put(PF_RAYO, F4(R.wo.x, R.wo.y, R.wo.z, R.tmax));
    c.put(PF_RAYD, R.wd, R.any ? kRayAny : L.stage == ST_PRIMARY ? kRayCamera : kRayBounce);
    c.put(PF_SEED, F4(__uint_as_float(L.seed.v[0]), __uint_as_float(L.seed.v[1]), __uint_as_float(L.seed.v[2]),
                      __uint_as_float(L.seed.v[3])));
    const uint32_t flags = L.stage | (L.chanceReflect ? 8u : 0u) | (L.back ? 16u : 0u) | (L.diel ? 32u : 0u) |
                           (L.hitReflect ? 64u : 0u) | (L.hitMetal ? 128u : 0u) | (L.neeLobe ? 256u : 0u);
    c.put(PF_STATE, F4(__int_as_float(L.pix), __uint_as_float(flags), __uint_as_float(L.i), __uint_as_float(L.b)));
    if (L.stage != ST_PRIMARY) c.put(PF_RC, L.rc);
    if (R.any && L.stage != ST_DIRECT) {   // the logic goes on from the vertex the ray left
        c.put(PF_VP, L.vs.P, L.vs.mat);
        c.put(PF_VN, L.vs.N, 0u);
        c.put(PF_DIR, L.dir, 0u);
    }
}

template <class Ctx>
__device__ __forceinline__ void load_path(const Ctx& c, Lane& L, PathRay& R) {
    const f4 o = c.get(PF_RAYO), d = c.get(PF_RAYD), h = c.get(PF_HIT), sd = c.get(PF_SEED), st = c.get(PF_STATE);
    R.wo = xyz(o); R.wd = xyz(d); R.tmax = o.w; R.any = __float_as_uint(d.w) == kRayAny;
    R.inst = __float_as_uint(h.x); R.prim = __float_as_uint(h.y); R.tri = __float_as_uint(h.z);
    R.hit = R.inst != 0xFFFFFFFFu;
    L.seed.v[0] = __float_as_uint(sd.x); L.seed.v[1] = __float_as_uint(sd.y);
    L.seed.v[2] = __float_as_uint(sd.z); L.seed.v[3] = __float_as_uint(sd.w);
    L.pix = __float_as_int(st.x);
    const uint32_t f = __float_as_uint(st.y);
    L.stage = f & 7u;
    L.chanceReflect = (f & 8u) != 0u; L.back = (f & 16u) != 0u; L.diel = (f & 32u) != 0u;
    L.hitReflect = (f & 64u) != 0u; L.hitMetal = (f & 128u) != 0u; L.neeLobe = (f & 256u) != 0u;
    L.i = __float_as_uint(st.z); L.b = __float_as_uint(st.w);
    L.rc = F4(1.0f, 1.0f, 1.0f, 1.0f);
    if (L.stage != ST_PRIMARY) L.rc = c.get(PF_RC);
    L.dir = R.wd;
    if (R.any && L.stage != ST_DIRECT) {
        const f4 p = c.get(PF_VP);
        L.vs.P = xyz(p);
        L.vs.mat = __float_as_uint(p.w);
        L.vs.N = xyz(c.get(PF_VN));
        L.dir = xyz(c.get(PF_DIR));
    }
}

// kNee: emissive-triangle NEE compiled in (GKRT_NEE_EMISSIVE with a non-empty table); the
// reference mode runs the instantiation without it.
//
// What bounds it: instruction issue with too few warps to cover it (1080p bricks: 301 warp
// instructions per ray at 16.3 of 32 lanes, 419 at 12.4 when a warp traced its 32 rays to the end
// before shading them all in registers; an issue in 42 % of the cycles, waits per issue for node loads and
// pool fields 2.6, fixed latencies 1.7, instruction fetch 1.5; 1.6 GB of pools through DRAM). So the code is kept small: one copy of the node
// test, of the finished rays' hand-over, of the probe lookup and of the sampled direction (3 % to 17 % of
// the pass). Trace pass in registers / on the pools / with one copy of each, ms: 1080p bricks 3.43 /
// 2.97 / 2.84, 4K city 91.9 / 51.0 / 48.7, textured 17.7 / 8.2 / 6.4, Cornell 256 x 256 0.164 / 0.146 /
// 0.134, 720p on the probe grid 1.98 / 1.25 / 1.16.
//
// Shared memory (dynamic): per-thread traversal stacks of stack_words entries (the scene's
// depth bound), the world rays in flight, then each warp's path lists. A stack no larger than the
// scene needs leaves the rest of the SM's 256 KB to L1, which serves the node fetches.
// kOneBlocks: pools of one warp's worth, blocks per SM (0: larger pools)
template <bool kNee, bool kTex, int kOneBlocks>
__global__ void __launch_bounds__(kPtThreads, kOneBlocks ? kOneBlocks : kPtBlocks) k_trace_pass(ShadeScene sc, GkrtFrameConstants fc, int W, int H,
                                                           int P, PixelImages im, unsigned long long* counters,
                                                           unsigned int* work, int stack_words, float4* pools,
                                                           uint32_t np) {
    constexpr bool kOne = kOneBlocks != 0;
    extern __shared__ uint32_t dyn_smem[];
    const int tid = threadIdx.x, warp = tid >> 5;
    const unsigned lane = tid & 31u;
    uint32_t* stack = dyn_smem + tid;
    float* wray = reinterpret_cast<float*>(dyn_smem + stack_words * kPtThreads) + tid;
    PathId* lists = reinterpret_cast<PathId*>(dyn_smem + (stack_words + kPoolRayWords) * kPtThreads) + (uint32_t)warp * 5u * np;
    float4* pool = pools + (size_t)(blockIdx.x * kPtWarps + warp) * warp_pool_size(PF_COUNT, np, kOne);
    float4* stash = pool + PF_COUNT * np + lane;
    Counters cn;
    cn.rays = 0; cn.fallbacks = 0; cn.retraces = 0; cn.nodes = 0; cn.tris = 0; cn.hits = 0;
    const int tiles_x = (W + 7) / 8, tiles_y = (H + 3) / 4;
    const unsigned total = (unsigned)tiles_x * (unsigned)tiles_y * 32u;
    PathList spare{lists + 4u * np, (int)np};      // paths without a pixel
    for (uint32_t k = lane; k < np; k += 32u) spare.l[k] = (PathId)k;
    PathList queue{lists + 3u * np, 0};
    DoneLists done{lists, np, {0, 0, 0}};
    if (!kOne) stash_empty(stash, sc.S);
    __syncwarp();
    bool exhausted = false;
    int live = 0;                                  // paths with a ray queued, in flight or finished
    for (;;) {
        // shading phase: the paths whose rays are finished, up to their next rays
        int take[3];
        const bool pure = done.largest() >= 32;
#pragma unroll
        for (int q = 0; q < 3; ++q) take[q] = pure ? done.n[q] & ~31 : done.n[q];
        const int n = take[0] + take[1] + take[2];
        live -= n;
        for (int k0 = 0; k0 < n; k0 += 32) {
            const int k = k0 + (int)lane;
            bool ray = false;
            uint32_t slot = 0;
            if (k < n) {
                slot = done.at(k, take);
                const Ctx<kOne> c{sc, fc, im, W, H, P, pool + slot, np, cn};
                Lane L;
                PathRay R;
                load_path(c, L, R);
                ray = advance<kNee, kTex>(L, R, c);
                if (ray) store_path(c, L, R);
            }
            __syncwarp();
            queue.add(ray, slot);
            spare.add(k < n && !ray, slot);
        }
        done.drop(take);
        // pixels into the spare paths, 32 at a time
        while (spare.n > 0 && !exhausted) {
            const int take = min(spare.n, 32);
            unsigned base = 0;
            if (lane == 0) base = atomicAdd(work, (unsigned)take);
            base = __shfl_sync(0xFFFFFFFFu, base, 0);
            const unsigned k = base + lane;
            exhausted = base + (unsigned)take >= total;
            bool ray = false;
            uint32_t slot = 0;
            if ((int)lane < take) {
                slot = spare.l[spare.n - take + (int)lane];
                const unsigned tile = k >> 5, in = k & 31u;
                const int x = (int)((tile % (unsigned)tiles_x) * 8u + (in & 7u));
                const int y = (int)((tile / (unsigned)tiles_x) * 4u + (in >> 3));
                ray = k < total && x < W && y < H;
                if (ray) {
                    const Ctx<kOne> c{sc, fc, im, W, H, P, pool + slot, np, cn};
                    Lane L;
                    PathRay R;
                    start_pixel(L, R, c, x, y);
                    L.i = 0; L.b = 0;
                    L.chanceReflect = L.back = L.diel = L.hitReflect = L.hitMetal = L.neeLobe = false;
                    store_path(c, L, R);
                }
            }
            spare.n -= take;
            __syncwarp();
            queue.add(ray, slot);
            spare.add((int)lane < take && !ray, slot);
            __syncwarp();
        }
        live += queue.n;
        if (live == 0) break;
        trace_queue<kOne>(sc.S, queue, done, pool, np, stash, wray, stack, stack_words, cn);
    }
    flush_counters(cn, counters);
}

// What bounds it: instruction issue and the latency of each ray's chain of nodes. 2 M incoherent rays
// of the 10 M-triangle city 2543 -> 1354 us (any-hit 2060 -> 853), of the bricks 1472 -> 943, of the
// Cornell box 680 -> 423; 1000 rays 35 -> 21 us. Before, one ray per thread over the 8-wide nodes
// with 72-word stacks, each warp waiting for its longest ray. 3 / 4 / 5 / 6 resident blocks: city 2 M
// 1375 / 1390 / 1354 / 1446, bricks 970 / 986 / 943 / 1001 us.
constexpr int kRqBlocks = 5;
__global__ void __launch_bounds__(kQueryThreads, kRqBlocks) k_trace_rays(SceneView S, const GkrtRay* rays, GkrtHit* hits,
                                                                         uint32_t n, uint32_t mode, uint32_t per, int cap,
                                                                         unsigned long long* counters) {
    extern __shared__ __align__(16) uint32_t rq_smem[];
    Counters cn;
    cn.rays = 0; cn.fallbacks = 0; cn.retraces = 0; cn.nodes = 0; cn.tris = 0; cn.hits = 0;
    query_rays(S, rays, hits, n, mode, per, cap, rq_smem, cn);
    flush_counters(cn, counters);
}

}  // namespace gk

using namespace gk;

// Paths per pool and the pools' size: as many paths per warp as the frame has pixels for, in whole
// warps, up to kPoolMax. A share that ends within a warp's worth is rounded up, so that every pixel starts at
// once though some warps get none, but below 128 down: 640 x 480 with 128 / 96 paths: bricks 632 / 619 us, Cornell
// 385 / 371, field of bricks 579 / 573 (textured 587 / 651, city 1705 / 1785); 700 x 400 with 128 / 96:
// 620 / 588. Above, 720 x 480 with 160 / 128: city 1885 / 1946, bricks 700 / 671.
static uint32_t paths_per_pool(uint32_t pixels, uint32_t warps) {
    const uint32_t share = pixels / std::max(1u, warps), want = (share < 128u ? share : share + 31u) / 32u * 32u;
    return std::max(32u, std::min(kPoolMax, want));
}
static bool one_warp_pools(uint32_t pixels, int num_sms) { return pixels / (uint32_t)num_sms <= kPtOneWarps * 32u; }
size_t gkrt_trace_pool_bytes(uint32_t pixels, int num_sms) {
    const size_t warps = std::min<size_t>((size_t)num_sms * kPtBlocks, (size_t)pixels / kPtThreads + 1u) * kPtWarps;
    const bool one = one_warp_pools(pixels, num_sms);
    const size_t paths = one ? 32u * warps : std::min<size_t>(warps * kPoolMax, (size_t)pixels + 32u * warps);
    return (paths * PF_COUNT + warps * warp_pool_size(0, 0, one)) * sizeof(float4);
}

cudaError_t gkrt_launch_trace_pass(const ShadeScene& sc, const GkrtFrameConstants& fc, int W, int H, int P,
                                   const PixelImages& im, unsigned long long* counters, unsigned int* work,
                                   int num_sms, int stack_words, bool textured, float4* pool, size_t pool_bytes,
                                   cudaStream_t st) {
    if (stack_words < 1 || stack_words > kQuadStackMax) return cudaErrorInvalidValue;
    const bool nee = fc.nee_mode == GKRT_NEE_EMISSIVE && sc.nemit > 0u;
    const bool tex = textured || (fc.has_sky && (fc.flags & GKRT_FRAME_SKY_TEXTURE));
    if (tex && !sc.tex) return cudaErrorInvalidValue;
    const size_t smem = (size_t)(stack_words + kPoolRayWords) * kPtThreads * 4u + pool_list_bytes(kPoolMax);
    using Kernel = void (*)(ShadeScene, GkrtFrameConstants, int, int, int, PixelImages, unsigned long long*, unsigned int*,
                            int, float4*, uint32_t);
#define GK_PASSES(nee, tex) {k_trace_pass<nee, tex, 0>, k_trace_pass<nee, tex, 2>, k_trace_pass<nee, tex, 3>}
    static const Kernel kernels[2][2][3] = {{GK_PASSES(false, false), GK_PASSES(false, true)},
                                            {GK_PASSES(true, false), GK_PASSES(true, true)}};
#undef GK_PASSES
    const uint32_t pixels = (uint32_t)W * (uint32_t)H;
    const uint32_t per_sm = pixels / (uint32_t)num_sms;
    const int one = per_sm <= 2u * kPtThreads ? 1 : one_warp_pools(pixels, num_sms) ? 2 : 0;
    const Kernel f = kernels[nee][tex][one];
    // resident blocks per SM of each instantiation and stack size, queried once per device
    static int occ[kMaxDevices][2][2][3][kQuadStackMax + 1] = {};
    const int dev = current_device_slot();
    if (dev < 0) return cudaErrorInvalidDevice;
    int* o = &occ[dev][nee][tex][one][stack_words];
    cudaError_t e = cudaSuccess;
    if (!*o) {
        const int most = (kQuadStackMax + kPoolRayWords) * kPtThreads * 4 + (int)pool_list_bytes(kPoolMax);   // the deepest trees a build accepts
        e = cudaFuncSetAttribute((const void*)f, cudaFuncAttributeMaxDynamicSharedMemorySize, most);
        if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(o, f, kPtThreads, smem);
        if (e != cudaSuccess) return e;
    }
    uint32_t blocks = (uint32_t)(num_sms * std::max(1, std::min(*o, kPtBlocks)));
    blocks = std::min(blocks, (pixels + kPtThreads - 1) / kPtThreads);
    const uint32_t np = one ? 32u : paths_per_pool(pixels, blocks * kPtWarps);
    if ((size_t)blocks * kPtWarps * warp_pool_size(PF_COUNT, np, one != 0) * sizeof(float4) > pool_bytes) return cudaErrorInvalidValue;
    e = cudaMemsetAsync(work, 0, sizeof(unsigned int), st);
    if (e != cudaSuccess) return e;
    f<<<blocks, kPtThreads, smem, st>>>(sc, fc, W, H, P, im, counters, work, stack_words, pool, np);
    return cudaGetLastError();
}

cudaError_t gkrt_launch_trace_rays(const SceneView& S, const GkrtRay* rays, GkrtHit* hits, uint32_t n,
                                   uint32_t mode, unsigned long long* counters, int stack_words, int num_sms,
                                   cudaStream_t st) {
    if (n == 0) return cudaSuccess;
    if (stack_words < 1 || stack_words > kQuadStackMax) return cudaErrorInvalidValue;
    static int occ[kMaxDevices][kQuadStackMax + 1] = {};
    const int dev = current_device_slot();
    if (dev < 0) return cudaErrorInvalidDevice;
    int* o = &occ[dev][stack_words];
    const size_t smem = query_smem(stack_words);
    if (!*o) {
        cudaError_t e = cudaFuncSetAttribute(k_trace_rays, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             (int)query_smem(kQuadStackMax));
        if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(o, k_trace_rays, kQueryThreads, smem);
        if (e != cudaSuccess) return e;
    }
    uint32_t blocks, per;
    query_grid(n, num_sms, *o, blocks, per);
    k_trace_rays<<<blocks, kQueryThreads, smem, st>>>(S, rays, hits, n, mode, per, stack_words, counters);
    return cudaGetLastError();
}
