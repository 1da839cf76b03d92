// k_adjoint.cu — differentiable rendering of the path-tracing estimator (path replay).
//
// No counterpart in the reference. The forward kernel evaluates the pass's estimator
// (FPathTracingRendererV2::Render / GetRayColor, assets/shaders/common/Shading.slang:1003-1184,
// reference NEE mode, no sun) for `spp` samples per pixel from the primary hit, and the
// composed linear radiance of the compose pass (diffuse x primary albedo + specular,
// Process.DenoiseJBF.comp.slang:147, without the filter). The backward kernel replays the
// same paths (same per-pixel RNG stream) and accumulates d loss / d material parameters:
//
//   albedo    every path is a product of albedo factors (the hit surface's albedo when the
//             bounce leaving the previous vertex was not a Schlick reflection, Shading.slang:
//             1053-1056; the primary albedo for metallic first bounces, :1159-1162; the
//             primary albedo of the remodulation) times the rest; d path / d factor k is the
//             product of the other factors and the rest (prefix x suffix, no division);
//   roughness the reference gives GGX-sampled bounces weight 1 and its roughness acts only
//             through the sampled direction. Sampling is detached here: the microfacet normal
//             m is drawn with roughness a_s and the bounce is weighted by p(m; a)/p(m; a_s),
//             where p is the density of the bounded VNDF sampler for a view along the
//             sampling axis (Eto and Tokuyoshi 2023; Const_Func.slang:310-340):
//                 p(m; a) = D(m; a) (axis . m) (1 + a^2),  D the GGX distribution.
//             At a = a_s the weight is exactly 1, so the value is the reference estimator's;
//             the gradient is the likelihood-ratio (score) term d log p / d a. The change of
//             the sampler's support with a is not differentiated.
//
// A pixel is a path of a warp's pool (gk_pool.cuh), its samples in sequence: every path runs its
// logic to the next ray, then the warp traces the rays of its pool. The backward pass records the
// current sample's factors and scores in the path's pool fields; at the sample's end every
// contribution is added to the FP64 sums in device memory, so that no FP32 sum of many terms is
// formed.
#include <algorithm>

#include "gk_pool.cuh"
#include "gk_shade.cuh"
#include "gkrt_internal.h"

namespace gk {

namespace {

// Resident blocks per SM (128 registers); 3 / 4 / 5 blocks took 19.9 / 17.8 / 16.6 ms forward and
// 20.1 / 18.6 / 18.5 backward with pools of 80 / 96 / 64 paths (4 blocks with 64: 16.5 / 17.5).
constexpr int kAdjBlocks = 4;
// Pools of one warp's worth of paths (kOne): at 3 blocks per SM up to 16 warps' worth of pixels per SM, at
// 4 up to 48. Forward and backward, us, pools of more / 3 / 4 blocks: 100 x 100 pixels at 16 samples 13953 /
// 10340 / 10755, 256 x 256 at 8 9811 / 7023 / 7706, 300 x 400 at 4 5866 / 5415 / 4618, 400 x 500 8798 /
// 7783 / 6959, 512 x 512 9670 / 11323 / 10217.
constexpr int kAdjOneWarps3 = 16, kAdjOneWarps4 = 48;
// Records of one sample: a factor per ray's hit and one for a metallic first bounce, a score per
// GGX bounce. The entry points take at most 16 bounces, a ray each.
constexpr int kMaxRays = 16;
constexpr int kMaxFactors = kMaxRays + 1;
constexpr int kMaxGgx = kMaxRays;

// A path's pool fields: its ray and answer, the RNG state, the throughput, the state word, the
// primary vertex (position and material; normal and bounce bound) and the two accumulators;
// backward also the product of the non-albedo multipliers, the albedo factors (rgb, material) and
// the scores (two records of material and score per field).
enum AdjField {
    AF_SEED = PF_FIRST_OWN, AF_RC, AF_STATE, AF_PP, AF_PN, AF_FC, AF_FR, AF_FORWARD_COUNT,
    AF_REST = AF_FORWARD_COUNT, AF_FAC, AF_GGX = AF_FAC + kMaxFactors, AF_BACKWARD_COUNT = AF_GGX + kMaxGgx / 2
};
template <bool kBackward>
constexpr uint32_t adj_fields() { return kBackward ? AF_BACKWARD_COUNT : AF_FORWARD_COUNT; }

enum AdjStage : uint32_t { AS_PRIMARY = 0, AS_FIRST = 1, AS_BOUNCE = 2 };

__device__ __forceinline__ float ggx_density_ratio_terms(float a, float c) {
    // a^2 (1 + a^2) / (c^2 (a^2 - 1) + 1)^2, the a-dependent part of p(m; a)
    const float a2 = a * a;
    const float q = fmaf_(c * c, a2 - 1.0f, 1.0f);
    return div_(a2 * (1.0f + a2), q * q);
}

__device__ __forceinline__ float ggx_score(float a, float c) {
    // d/da log p(m; a) = 2/a + 2a/(1 + a^2) - 4 a c^2 / (c^2 (a^2 - 1) + 1)
    const float a2 = a * a, c2 = c * c;
    return (div_(2.0f, a) + div_(2.0f * a, 1.0f + a2)) - div_((4.0f * a) * c2, fmaf_(c2, a2 - 1.0f, 1.0f));
}

// Camera ray of FHardwarePrimaryRayCaster (Shading.slang:286-304), as start_pixel.
__device__ void camera_ray(const GkrtFrameConstants& fc, int x, int y, int W, int H, Rng& seed, f3& o, f3& d) {
    float uvx = fmaf_(div_((float)x, (float)W), 2.0f, -1.0f);
    float uvy = fmaf_(div_((float)y, (float)H), 2.0f, -1.0f);
    if (fc.taa) {
        const uint32_t hi = fc.total_frames % 8u;
        uvx = uvx + div_(c_halton[2 * hi] - 0.5f, (float)W);
        uvy = uvy + div_(c_halton[2 * hi + 1] - 0.5f, (float)H);
    }
    const f2 disk = unit_disk(seed);
    const float ha = div_(fc.aperture, 2.0f);
    const float offx = ha * disk.x, offy = ha * disk.y;
    const f4 origin = mat4v(fc.model_view_inverse, F4(offx, offy, 0.0f, 1.0f));
    const f4 target = mat4v(fc.projection_inverse, F4(uvx, uvy, 1.0f, 1.0f));
    const f3 tn = normalize3(F3(fmaf_(target.x, fc.focus_distance, -offx), fmaf_(target.y, fc.focus_distance, -offy),
                                target.z * fc.focus_distance));
    const f4 direction = mat4v(fc.model_view_inverse, F4(tn.x, tn.y, tn.z, 0.0f));
    o = xyz(origin);
    d = xyz(direction);
}

struct AdjArgs {
    int W, H;
    uint32_t spp;
    const float* sample_rough;   // per material, or null: sample with the material's own
    float4* image;               // forward
    const float4* dimage;        // backward
    double* g_alb;
    double* g_rough;
};

template <bool kOne>
struct AdjPath {
    float4* p;        // field 0
    uint32_t np;      // stride between fields
    __device__ f4 get(int f) const {
        const float4 v = pool_get<kOne>(p + (uint32_t)f * np);
        return F4(v.x, v.y, v.z, v.w);
    }
    __device__ void put(int f, f4 v) const {
        pool_put<kOne>(p + (uint32_t)f * np, make_float4(v.x, v.y, v.z, v.w));
    }
    __device__ void put(int f, f3 v, uint32_t w) const { put(f, F4(v.x, v.y, v.z, __uint_as_float(w))); }
    __device__ float2* ggx(int k) const {
        return reinterpret_cast<float2*>(p + (uint32_t)(AF_GGX + (k >> 1)) * np) + (k & 1);
    }
};

__device__ __forceinline__ void add_grad(double* g, float v) {
    if (v != 0.0f) atomicAdd(g, (double)v);
}

// Runs a path on the answer of its ray, up to its next ray (true) or the end of its pixel (false):
// FPathTracingRendererV2::Render and GetRayColor (Shading.slang:1003-1184) with detached GGX
// sampling and, backward, the sample's records.
template <bool kBackward, class AdjPath>
__device__ __forceinline__ bool adj_advance(const ShadeScene& sc, const GkrtFrameConstants& fc, const AdjArgs& a,
                                            const AdjPath& c, Counters& cn) {
    const f4 ro = c.get(PF_RAYO), rd = c.get(PF_RAYD), h = c.get(PF_HIT), sd = c.get(AF_SEED), state = c.get(AF_STATE);
    Rng seed;
    seed.v[0] = __float_as_uint(sd.x); seed.v[1] = __float_as_uint(sd.y);
    seed.v[2] = __float_as_uint(sd.z); seed.v[3] = __float_as_uint(sd.w);
    const int pix = __float_as_int(state.x);
    // stage (2 bits), chanceReflect, back, diel, hitReflect, hitMetal, factors (5 bits), scores (5 bits)
    uint32_t fl = __float_as_uint(state.y);
    const uint32_t stage = fl & 3u;
    uint32_t i = __float_as_uint(state.z), b = __float_as_uint(state.w);
    bool chanceReflect = (fl & 4u) != 0u, back = (fl & 8u) != 0u, diel = (fl & 16u) != 0u;
    bool hitReflect = (fl & 32u) != 0u, hitMetal = (fl & 64u) != 0u;
    int nf = (int)((fl >> 8) & 31u), ng = (int)((fl >> 16) & 31u);
    const bool hit = __float_as_uint(h.x) != 0xFFFFFFFFu;
    const uint32_t nm = sc.nmat;
    f4 rc = F4(1.0f, 1.0f, 1.0f, 1.0f), rest = F4(1.0f, 1.0f, 1.0f, 1.0f);
    if (stage != AS_PRIMARY) {
        rc = c.get(AF_RC);
        if (kBackward) rest = c.get(AF_REST);
    }
    Vtx v;
    if (hit) v = hit_vertex(sc, xyz(ro), xyz(rd), __float_as_uint(h.x), __float_as_uint(h.y), __float_as_uint(h.z));
    bool need_begin = false, need_pre = false, need_end = false, pre_first = false, done = false;
    f4 out = F4(0.0f, 0.0f, 0.0f, 1.0f);

    if (stage == AS_PRIMARY) {
        done = true;
        if (!hit) {
            const f4 s = sky(fc);
            out = F4(s.x, s.y, s.z, 1.0f);
        } else {
            const MatV pm = load_mat(sc, v.mat);
            if (pm.model != GKRT_MAT_DIELECTRIC) v.P = fma3(normalize3(xyz(rd)), -0.03f, v.P);
            if (pm.model == GKRT_MAT_DIFFUSE_LIGHT) {
                out = F4(pm.diffuse.x, pm.diffuse.y, pm.diffuse.z, 1.0f);
            } else {
                const bool pdiel = pm.model == GKRT_MAT_DIELECTRIC;
                c.put(AF_PP, v.P, v.mat);
                c.put(AF_PN, v.N, (pdiel ? fc.max_number_of_bounces : fc.number_of_bounces) | (pdiel ? 0x80000000u : 0u));
                c.put(AF_FC, F4(0.0f, 0.0f, 0.0f, 0.0f));
                c.put(AF_FR, F4(0.0f, 0.0f, 0.0f, 0.0f));
                i = 0;
                need_begin = true;
                done = false;
            }
        }
    } else {
        // after the ray (Shading.slang:1039-1081)
        bool term = true;
        if (hit) {
            const MatV hm = load_mat(sc, v.mat);
            if (hm.model == GKRT_MAT_DIFFUSE_LIGHT || !chanceReflect) {
                rc = rc * hm.diffuse;
                if (kBackward && nf < kMaxFactors) c.put(AF_FAC + nf++, xyz(hm.diffuse), v.mat);
            }
            if (back && !diel) {
                rc = F4(0.5f, 0.5f, 0.5f, 0.0f);   // constant: no parameter reaches this path
                nf = 0;
                ng = 0;
                rest = rc;
            } else {
                term = hm.model == GKRT_MAT_DIFFUSE_LIGHT;
            }
        } else {
            const f4 s = sky(fc);
            rc = rc * s;
            rest = rest * s;
        }
        need_end = term;
        if (!term) {
            const uint32_t loop = __float_as_uint(c.get(AF_PN).w);
            const uint32_t maxB = loop & 0x7FFFFFFFu;
            const bool pdiel = (loop >> 31) != 0u;
            bool probe = false;
            if (stage == AS_FIRST) {
                if (fc.fast_gather && !pdiel) {
                    probe = true;
                } else {
                    b = 1;
                    need_end = !(b < maxB);
                }
            } else {
                const bool early = !pdiel && rnd1(seed) < 0.5f;
                probe = b == maxB - 1u || early;
                if (!probe) ++b;
            }
            if (probe) {
                const f4 pt = probe_term(sc, v.P, v.N);
                rc = rc * pt;
                rest = rest * pt;
                need_end = true;
            }
            need_pre = !need_end;
        }
    }

    // the sample's end (Shading.slang:1159-1176): its value, and backward its gradients
    if (need_end) {
        const f4 pp = c.get(AF_PP);
        const uint32_t pmat = __float_as_uint(pp.w);
        const f4 ap = load_mat(sc, pmat).diffuse;
        if (hitMetal) {
            rc = rc * ap;
            if (kBackward && nf < kMaxFactors) c.put(AF_FAC + nf++, xyz(ap), pmat);
        }
        const int acc = hitReflect ? AF_FR : AF_FC;
        if (!kBackward) c.put(acc, c.get(acc) + rc);
        if (kBackward) {
            const float4 gi = __ldg(&a.dimage[pix]);
            const f4 g = F4(gi.x, gi.y, gi.z, 0.0f);
            const float inv_spp = div_(1.0f, (float)a.spp);
            // upstream of this path's value: remodulated (diffuse) or not (specular)
            const f4 u = hitReflect ? g * inv_spp : (g * ap) * inv_spp;
            if (!hitReflect) {
                const uint32_t mp = pmat < nm ? pmat : nm - 1u;
                add_grad(&a.g_alb[3 * mp + 0], (g.x * rc.x) * inv_spp);
                add_grad(&a.g_alb[3 * mp + 1], (g.y * rc.y) * inv_spp);
                add_grad(&a.g_alb[3 * mp + 2], (g.z * rc.z) * inv_spp);
            }
            // d path / d factor k = prefix(k) * suffix(k) * rest
            f4 pre = F4(1.0f, 1.0f, 1.0f, 1.0f);
            for (int k = 0; k < nf; ++k) {
                f4 suf = rest;
                for (int j = k + 1; j < nf; ++j) suf = suf * c.get(AF_FAC + j);
                const f4 fk = c.get(AF_FAC + k);
                const f4 dk = (pre * suf) * u;
                const uint32_t mk = min(__float_as_uint(fk.w), nm - 1u);
                add_grad(&a.g_alb[3 * mk + 0], dk.x);
                add_grad(&a.g_alb[3 * mk + 1], dk.y);
                add_grad(&a.g_alb[3 * mk + 2], dk.z);
                pre = pre * fk;
            }
            const float uc = fmaf_(u.z, rc.z, fmaf_(u.y, rc.y, u.x * rc.x));
            for (int k = 0; k < ng; ++k) {
                const float2 r = __ldcg(c.ggx(k));
                add_grad(&a.g_rough[min(__float_as_uint(r.x), nm - 1u)], uc * r.y);
            }
        }
        if (++i < a.spp) {
            need_begin = true;
        } else {
            done = true;
            if (!kBackward) {
                f4 fcol = c.get(AF_FC), frefl = c.get(AF_FR);
                const float fs = (float)a.spp;
                fcol = F4(div_(fcol.x, fs), div_(fcol.y, fs), div_(fcol.z, fs), div_(fcol.w, fs));
                frefl = F4(div_(frefl.x, fs), div_(frefl.y, fs), div_(frefl.z, fs), div_(frefl.w, fs));
                out = F4(fmaf_(fcol.x, ap.x, frefl.x), fmaf_(fcol.y, ap.y, frefl.y), fmaf_(fcol.z, ap.z, frefl.z), 1.0f);
            }
        }
    }
    if (done) {
        if (!kBackward) a.image[pix] = make_float4(out.x, out.y, out.z, out.w);
        return false;
    }

    // a sample's start
    f3 dir = xyz(rd);
    if (need_begin) {
        const f4 eye = mat4v(fc.model_view_inverse, F4(0.0f, 0.0f, 0.0f, 1.0f));
        const f4 pp = c.get(AF_PP);
        v.P = xyz(pp);
        v.N = xyz(c.get(AF_PN));
        v.mat = __float_as_uint(pp.w);
        dir = normalize3(v.P - xyz(eye));
        rc = F4(1.0f, 1.0f, 1.0f, 1.0f);
        rest = rc;
        nf = 0;
        ng = 0;
        hitReflect = false;
        hitMetal = false;
        pre_first = true;
    }

    // GetRayColor up to its trace (Shading.slang:1007-1039), GGX bounces weighted and scored
    const MatV mat = load_mat(sc, v.mat);
    diel = mat.model == GKRT_MAT_DIELECTRIC;
    const float startPosOffset = diel ? 0.0f : 1.0f;
    const float dotValue = dot3(dir, v.N);
    back = dotValue > 0.0f;
    const f3 outward = back ? -v.N : v.N;
    const float niOverNt = back ? mat.ri2 : div_(1.0f, mat.ri2);
    const float cosine = dotValue > 0.0f ? mat.ri * dotValue : -dotValue;
    const float reflectProb = schlick(cosine, mat.ri);
    chanceReflect = rnd1(seed) < reflectProb;
    const bool chanceMetal = rnd1(seed) < mat.metal;
    const bool chanceGGX = chanceReflect || chanceMetal;
    f3 tdir;
    float ggx_c = 0.0f, a_s = 0.0f;
    if (chanceGGX) {
        const f3 axis = reflect3(dir, outward);
        const uint32_t mi = v.mat < nm ? v.mat : nm - 1u;
        const float fs = a.sample_rough ? __ldg(&a.sample_rough[mi]) : mat.fuzz;
        const float r = sqrt_(fs);
        a_s = r * r;
        tdir = ggx_sample(seed, r, axis);
        ggx_c = dot3(axis, tdir);
    } else {
        tdir = align_normal(hemisphere_cos(seed), outward);
    }
    if (pre_first) { hitReflect = chanceGGX; hitMetal = chanceMetal; }
    const bool refracted = diel && !chanceReflect;
    if (refracted) tdir = refract3(dir, outward, niOverNt);
    if (chanceGGX && !refracted && a_s > 1e-6f) {
        const float re = sqrt_(mat.fuzz);
        const float a_e = re * re;
        if (a_e != a_s) {
            const float w = div_(ggx_density_ratio_terms(a_e, ggx_c), ggx_density_ratio_terms(a_s, ggx_c));
            rc = rc * w;
            rest = rest * w;
        }
        if (kBackward && ng < kMaxGgx) {
            __stcg(c.ggx(ng), make_float2(__uint_as_float(v.mat), a_e > 1e-6f ? ggx_score(a_e, ggx_c) : 0.0f));
            ++ng;
        }
    }
    const f3 org = fma3(v.N, 0.001f * startPosOffset, v.P);
    ++cn.rays;
    c.put(PF_RAYO, F4(org.x, org.y, org.z, 1000.0f));
    c.put(PF_RAYD, tdir, kRayBounce);
    c.put(AF_SEED, F4(__uint_as_float(seed.v[0]), __uint_as_float(seed.v[1]), __uint_as_float(seed.v[2]),
                      __uint_as_float(seed.v[3])));
    c.put(AF_RC, rc);
    if (kBackward) c.put(AF_REST, rest);
    fl = (pre_first ? AS_FIRST : AS_BOUNCE) | (chanceReflect ? 4u : 0u) | (back ? 8u : 0u) | (diel ? 16u : 0u) |
         (hitReflect ? 32u : 0u) | (hitMetal ? 64u : 0u) | ((uint32_t)nf << 8) | ((uint32_t)ng << 16);
    c.put(AF_STATE, F4(state.x, __uint_as_float(fl), __uint_as_float(i), __uint_as_float(b)));
    return true;
}

// Persistent warps over the frame's pixels (row-major, 32 at a time). What bounds it: as the rt pass,
// instruction issue; one thread per pixel, every warp waiting for its longest path at each ray of
// each sample, took 40.7 ms forward and 51 backward at 512 x 512 and 16 samples; now 16.5 and 17.5.
// kOneBlocks: pools of one warp's worth, blocks per SM (0: larger pools)
template <bool kBackward, int kOneBlocks>
__global__ void __launch_bounds__(kPoolThreads, kOneBlocks ? kOneBlocks : kAdjBlocks) k_adjoint(ShadeScene sc, GkrtFrameConstants fc, AdjArgs a,
                                                                      unsigned long long* counters, unsigned int* work,
                                                                      int stack_words, float4* pools, uint32_t np) {
    constexpr bool kOne = kOneBlocks != 0;
    extern __shared__ uint32_t adj_smem[];
    const int tid = threadIdx.x, warp = tid >> 5;
    const unsigned lane = tid & 31u;
    uint32_t* stack = adj_smem + tid;
    float* wray = reinterpret_cast<float*>(adj_smem + stack_words * kPoolThreads) + tid;
    PathId* lists = reinterpret_cast<PathId*>(adj_smem + (stack_words + kPoolRayWords) * kPoolThreads) +
                    (uint32_t)warp * 5u * np;
    float4* pool = pools + (size_t)(blockIdx.x * kPoolWarps + warp) * warp_pool_size(adj_fields<kBackward>(), np, kOne);
    float4* stash = pool + adj_fields<kBackward>() * np + lane;
    Counters cn;
    cn.rays = 0; cn.fallbacks = 0; cn.retraces = 0; cn.nodes = 0; cn.tris = 0; cn.hits = 0;
    const unsigned total = (unsigned)a.W * (unsigned)a.H;
    PathList spare{lists + 4u * np, (int)np};
    for (uint32_t k = lane; k < np; k += 32u) spare.l[k] = (PathId)k;
    PathList queue{lists + 3u * np, 0};
    DoneLists done{lists, np, {0, 0, 0}};
    if (!kOne) stash_empty(stash, sc.S);
    __syncwarp();
    bool exhausted = false;
    int live = 0;
    for (;;) {
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
                ray = adj_advance<kBackward>(sc, fc, a, AdjPath<kOne>{pool + slot, np}, cn);
            }
            __syncwarp();
            queue.add(ray, slot);
            spare.add(k < n && !ray, slot);
        }
        done.drop(take);
        while (spare.n > 0 && !exhausted) {
            const int want = min(spare.n, 32);
            unsigned base = 0;
            if (lane == 0) base = atomicAdd(work, (unsigned)want);
            base = __shfl_sync(0xFFFFFFFFu, base, 0);
            const unsigned pix = base + lane;
            exhausted = base + (unsigned)want >= total;
            bool ray = false;
            uint32_t slot = 0;
            if ((int)lane < want) {
                slot = spare.l[spare.n - want + (int)lane];
                ray = pix < total;
                if (ray) {
                    const int x = (int)(pix % (unsigned)a.W), y = (int)(pix / (unsigned)a.W);
                    Rng seed;
                    seed.v[0] = (uint32_t)x; seed.v[1] = (uint32_t)y; seed.v[2] = fc.total_frames; seed.v[3] = 0u;
                    f3 o, d;
                    camera_ray(fc, x, y, a.W, a.H, seed, o, d);
                    ++cn.rays;
                    const AdjPath<kOne> c{pool + slot, np};
                    c.put(PF_RAYO, F4(o.x, o.y, o.z, 1000.0f));
                    c.put(PF_RAYD, d, kRayCamera);
                    c.put(AF_SEED, F4(__uint_as_float(seed.v[0]), __uint_as_float(seed.v[1]),
                                      __uint_as_float(seed.v[2]), __uint_as_float(seed.v[3])));
                    c.put(AF_STATE, F4(__int_as_float((int)pix), __uint_as_float((uint32_t)AS_PRIMARY), 0.0f, 0.0f));
                }
            }
            spare.n -= want;
            __syncwarp();
            queue.add(ray, slot);
            spare.add((int)lane < want && !ray, slot);
            __syncwarp();
        }
        live += queue.n;
        if (live == 0) break;
        trace_queue<kOne>(sc.S, queue, done, pool, np, stash, wray, stack, stack_words, cn);
    }
    // ray counters: warp sums, one atomic per warp
    unsigned long long r = cn.rays;
    for (int o2 = 16; o2 > 0; o2 >>= 1) r += __shfl_down_sync(0xFFFFFFFFu, r, o2);
    if ((tid & 31) == 0 && r) atomicAdd(&counters[0], r);
}

// Material parameters from device arrays: diffuse rgb and fuzziness of materials
// [first, first + count).
__global__ void k_set_params(GkrtMaterial* mats, const float* alb, const float* rough, uint32_t first,
                             uint32_t count) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= count) return;
    GkrtMaterial& m = mats[first + i];
    if (alb) {
        m.diffuse[0] = alb[3 * i];
        m.diffuse[1] = alb[3 * i + 1];
        m.diffuse[2] = alb[3 * i + 2];
    }
    if (rough) m.fuzziness = rough[i];
}

}  // namespace

}  // namespace gk

using namespace gk;

cudaError_t gkrt_launch_adjoint(const ShadeScene& sc, const GkrtFrameConstants& fc, int W, int H, uint32_t spp,
                                const float* sample_rough, float4* image, const float4* dimage, double* g_alb,
                                double* g_rough, unsigned long long* counters, int stack_words, int num_sms,
                                cudaMemPool_t mem, cudaStream_t st) {
    if (stack_words < 1 || stack_words > kQuadStackMax) return cudaErrorInvalidValue;
    using Kernel = void (*)(ShadeScene, GkrtFrameConstants, AdjArgs, unsigned long long*, unsigned int*, int, float4*,
                            uint32_t);
    static const Kernel kernels[2][3] = {{k_adjoint<false, 0>, k_adjoint<false, 3>, k_adjoint<false, 4>},
                                         {k_adjoint<true, 0>, k_adjoint<true, 3>, k_adjoint<true, 4>}};
    const uint32_t pixels = (uint32_t)W * (uint32_t)H;
    const uint32_t sm_warps = pixels / (uint32_t)num_sms / 32u;
    const int one = sm_warps < (uint32_t)kAdjOneWarps3 ? 1 : sm_warps < (uint32_t)kAdjOneWarps4 ? 2 : 0;
    const Kernel f = kernels[dimage != nullptr][one];
    const uint32_t fields = dimage ? adj_fields<true>() : adj_fields<false>();
    const size_t smem = (size_t)(stack_words + kPoolRayWords) * kPoolThreads * 4u + pool_list_bytes(kPoolMax);
    static int occ[kMaxDevices][2][3][kQuadStackMax + 1] = {};
    const int dev = current_device_slot();
    if (dev < 0) return cudaErrorInvalidDevice;
    int* o = &occ[dev][dimage ? 1 : 0][one][stack_words];
    cudaError_t e = cudaSuccess;
    if (!*o) {
        const int most = (kQuadStackMax + kPoolRayWords) * kPoolThreads * 4 + (int)pool_list_bytes(kPoolMax);
        e = cudaFuncSetAttribute((const void*)f, cudaFuncAttributeMaxDynamicSharedMemorySize, most);
        if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(o, f, kPoolThreads, smem);
        if (e != cudaSuccess) return e;
    }
    uint32_t blocks = (uint32_t)(num_sms * std::max(1, std::min(*o, kAdjBlocks)));
    blocks = std::min(blocks, (pixels + kPoolThreads - 1) / kPoolThreads);
    const uint32_t warps = blocks * kPoolWarps;
    // A pixel's samples are a long chain of rays: pools of two thirds of a warp's share of the pixels
    // leave the rest to the warps that end early (512 x 512 at 16 samples, a share of 107: pools of
    // 32 / 64 / 96 paths 21.2 / 16.5 / 17.8 ms forward).
    const uint32_t np = one ? 32u : std::max(32u, std::min(kPoolMax, pixels / warps * 2u / 3u / 32u * 32u));
    // scratch of this call alone (calls may overlap on several streams): the pools, then the pixel counter
    const size_t bytes = (size_t)warps * warp_pool_size(fields, np, one != 0) * sizeof(float4);
    float4* pools = nullptr;
    e = cudaMallocFromPoolAsync((void**)&pools, bytes + 16u, mem, st);
    if (e != cudaSuccess) return e;
    unsigned int* work = reinterpret_cast<unsigned int*>(reinterpret_cast<uint8_t*>(pools) + bytes);
    e = cudaMemsetAsync(work, 0, sizeof(unsigned int), st);
    if (e == cudaSuccess) {
        const AdjArgs a{W, H, spp, sample_rough, image, dimage, g_alb, g_rough};
        f<<<blocks, kPoolThreads, smem, st>>>(sc, fc, a, counters, work, stack_words, pools, np);
        e = cudaGetLastError();
    }
    const cudaError_t ef = cudaFreeAsync(pools, st);
    return e == cudaSuccess ? ef : e;
}

cudaError_t gkrt_launch_set_params(GkrtMaterial* mats, const float* alb, const float* rough, uint32_t first,
                                   uint32_t count, cudaStream_t st) {
    if (count == 0) return cudaSuccess;
    k_set_params<<<(count + 127) / 128, 128, 0, st>>>(mats, alb, rough, first, count);
    return cudaGetLastError();
}
