// k_probes.cu — ambient-cube probe grid: voxelization and bake on the GPU (sm_103a).
//
// The probe grid (192 x 48 x 192 probes, 0.25 m apart, AmbientCube.slang:12-15) feeds the
// path termination of the rt pass (probe_term). Two kernels fill it:
//   k_probe_voxelize  the distance data of every probe: six axis rays and, in open space, six
//                     diagonal rays, as the reference's CPU voxelizer does with tinybvh
//                     (VoxelizeCube / InsideGeometry / DetectDistance,
//                     src/Assets/CPUAccelerationStructure.cpp:70-160);
//   k_bake_*          one bake step of a slice of probes (Bake.HwAmbientCube.comp.slang:1-19,
//                     FGpuProbeGenerator::RenderAmbientCubeOnly and FaceTask,
//                     AmbientCube.slang:477-553, 656-690): per face 16 rays over a jittered
//                     4 x 4 grid, the bounce light of their hits from the probes around them,
//                     the sky, light 0 and the sun, blended into the packed colours with
//                     weight 1/8. Three kernels: the slice's surface probes are listed; persistent
//                     warps trace every ray of theirs (the ray queries' schedule) and keep its
//                     light; eight lanes per probe, six of them a face each, sum the rays' light in
//                     order and blend it in.
// The bake reads the neighbour probes it interpolates as they were before the step, so results
// do not depend on the order in which probes are updated (the reference reads and writes one
// buffer concurrently): the rays are all traced before the first probe is written, and steps
// of more probes than one batch read a snapshot of the grid.
#include <algorithm>

#include "gk_query.cuh"
#include "gk_shade.cuh"
#include "gkrt_internal.h"

namespace gk {

namespace {

constexpr int kVoxThreads = 128;
constexpr int kBakeThreads = 128;
constexpr uint32_t kFaceRays = 16;     // rays of a face; light 0 and the sun may add one each
constexpr float kCubeUnit = 0.25f;
constexpr float kFastMaxTrace = 20.0f;          // FAST_MAX_TRACE_DISTANCE, Shading.slang:16
constexpr float kOcclusionMax = 1000.0f;        // PT_MAX_TRACE_DISTANCE of TraceOcclusion
constexpr float kInvSqrt3 = 0.577350269f;

__constant__ float c_grid4x4[32] = {-0.75f, -0.75f, -0.25f, -0.75f, 0.25f, -0.75f, 0.75f, -0.75f,
                                    -0.75f, -0.25f, -0.25f, -0.25f, 0.25f, -0.25f, 0.75f, -0.25f,
                                    -0.75f, 0.25f,  -0.25f, 0.25f,  0.25f, 0.25f,  0.75f, 0.25f,
                                    -0.75f, 0.75f,  -0.25f, 0.75f,  0.25f, 0.75f,  0.75f, 0.75f};
__constant__ float c_grid3x3[18] = {-0.667f, -0.667f, 0.0f, -0.667f, 0.667f, -0.667f, -0.667f, 0.0f, 0.0f,
                                    0.0f,    0.667f,  0.0f, -0.667f, 0.667f, 0.0f,    0.667f, 0.667f, 0.667f};

// Warp-aggregated flush of the ray counters (per-pass slots 0-5, total rays in slot 6).
__device__ __forceinline__ void flush_ray_counters(const Counters& c, unsigned long long* out) {
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

GK_D f3 probe_origin(uint32_t g) {
    const uint32_t y = g / (uint32_t)(kProbeXY * kProbeXY);
    const uint32_t z = (g - y * (uint32_t)(kProbeXY * kProbeXY)) / (uint32_t)kProbeXY;
    const uint32_t x = g - y * (uint32_t)(kProbeXY * kProbeXY) - z * (uint32_t)kProbeXY;
    return F3((float)x * kCubeUnit + kProbeOffX, (float)y * kCubeUnit + kProbeOffY, (float)z * kCubeUnit + kProbeOffZ);
}

GK_D f3 face_basis(int f) {   // +Y, -Y, +X, -X, +Z, -Z (the order of RenderAmbientCubeOnly)
    const float s = (f & 1) ? -1.0f : 1.0f;
    return f < 2 ? F3(0.0f, s, 0.0f) : (f < 4 ? F3(s, 0.0f, 0.0f) : F3(0.0f, 0.0f, s));
}

struct ProbeHit {
    bool hit, back;
    float t;
    uint32_t mat;
};

// Closest hit over [EPS, tmax]: its float t, material, whether the ray met the triangle's
// back (object-space face normal cross(v1 - v0, v2 - v1), CPUAccelerationStructure.cpp:193-196).
GK_D ProbeHit probe_trace(const ShadeScene& sc, f3 o, f3 d, float tmax, uint32_t* stk, int stride, Counters& cn) {
    ProbeHit r;
    r.hit = false; r.back = false; r.t = 0.0f; r.mat = 0u;
    ++cn.rays;
    const TraceOut t = traverse_wide<kClosest>(sc.S, o, d, kTmin, tmax, stk, stride, cn);
    if (!t.hit) return r;
    r.hit = true;
    const HitShade h = hit_shade(sc.S, o, d, t.inst, t.tri);
    r.t = h.t;
    const DevInst* ip = sc.S.inst + t.inst;
    const uint32_t ioff = __ldg(&ip->index_offset) + 3u * t.prim, voff = __ldg(&ip->vertex_offset);
    r.mat = __ldg(&sc.inst_mat[16u * t.inst + (__ldg(&sc.slots[__ldg(&sc.indices[ioff]) + voff]) & 15u)]);
    const f3 v0 = tri_v(sc.S.tris, t.tri, 0), v1 = tri_v(sc.S.tris, t.tri, 1), v2 = tri_v(sc.S.tris, t.tri, 2);
    const f3 a = v1 - v0, b = v2 - v1;
    const f3 n = F3(fmaf_(a.y, b.z, -(a.z * b.y)), fmaf_(a.z, b.x, -(a.x * b.z)), fmaf_(a.x, b.y, -(a.y * b.x)));
    float w[12];
    load_winv(ip, w);
    const f3 dl = xvector(w, d);
    r.back = fmaf_(n.z, dl.z, fmaf_(n.y, dl.y, n.x * dl.x)) > 0.0f;
    return r;
}

GK_D uint32_t pack10(f4 c) {   // packRGB10A2 (AmbientCube.slang:59-69), MAX_ILLUMINANCE 512
    const float r = mn(mx(c.x * 0.001953125f, 0.0f), 1.0f), g = mn(mx(c.y * 0.001953125f, 0.0f), 1.0f);
    const float b = mn(mx(c.z * 0.001953125f, 0.0f), 1.0f), a = mn(mx(c.w * 0.001953125f, 0.0f), 1.0f);
    return (uint32_t)(r * 1023.0f) | ((uint32_t)(g * 1023.0f) << 10) | ((uint32_t)(b * 1023.0f) << 20) |
           ((uint32_t)(a * 3.0f) << 30);
}

GK_D float lerpf_(float a, float b, float t) { return fmaf_(t, b - a, a); }

// sampleAmbientCubeHL2_DI (AmbientCube.slang:127-150): the direct colours only.
GK_D f4 cube_sample_di(const uint32_t* cube, f3 n) {
    const float wx = mx(n.x, 0.0f), wnx = mx(-n.x, 0.0f), wy = mx(n.y, 0.0f), wny = mx(-n.y, 0.0f);
    const float wz = mx(n.z, 0.0f), wnz = mx(-n.z, 0.0f);
    const float sum = ((((wx + wnx) + wy) + wny) + wz) + wnz;
    // of each pair of directions only the one the normal faces has a weight
    f4 col = F4(0.0f, 0.0f, 0.0f, 0.0f);
    col = col + unpack10(__ldg(&cube[n.x > 0.0f ? 10 : 11])) * (n.x > 0.0f ? wx : wnx);
    col = col + unpack10(__ldg(&cube[n.y > 0.0f ? 8 : 9])) * (n.y > 0.0f ? wy : wny);
    col = col + unpack10(__ldg(&cube[n.z > 0.0f ? 6 : 7])) * (n.z > 0.0f ? wz : wnz);
    return col * (sum > 0.0f ? div_(1.0f, sum) : 1.0f);
}

// interpolateAmbientCubesV2<DIAmbientCubeSampler> (AmbientCube.slang:290-382) over the snapshot.
GK_D f4 probe_di(const uint32_t* cubes, const uint32_t* voxels, f3 p, f3 n) {
    const float npx = (p.x - kProbeOffX) * 4.0f, npy = (p.y - kProbeOffY) * 4.0f, npz = (p.z - kProbeOffZ) * 4.0f;
    if (!(npx >= 0.0f) || !(npy >= 0.0f) || !(npz >= 0.0f) || npx > (float)(kProbeXY - 2) ||
        npy > (float)(kProbeZ - 2) || npz > (float)(kProbeXY - 2))
        return F4(0.0f, 0.0f, 0.0f, 1.0f);
    const float fx = floorf(npx), fy = floorf(npy), fz = floorf(npz);
    const int bx = (int)fx, by = (int)fy, bz = (int)fz;
    const float frx = npx - fx, fry = npy - fy, frz = npz - fz;
    float tw = 0.0f;
    f4 res = F4(0.0f, 0.0f, 0.0f, 0.0f);
    for (int i = 0; i < 8; ++i) {
        const int ox = i & 1, oy = (i >> 1) & 1, oz = (i >> 2) & 1;
        const size_t id = (size_t)(by + oy) * kProbeXY * kProbeXY + (size_t)(bz + oz) * kProbeXY + (size_t)(bx + ox);
        const uint32_t u0 = __ldg(&voxels[id * 4 + 2]), u1 = __ldg(&voxels[id * 4 + 3]);
        const float d0y = div255((float)((u0 >> 8) & 0xFFu));
        if (d0y < 0.01f) continue;
        const float d0z = div255((float)((u0 >> 16) & 0xFFu)), d0w = div255((float)((u0 >> 24) & 0xFFu));
        const float d1x = div255((float)(u1 & 0xFFu)), d1y = div255((float)((u1 >> 8) & 0xFFu));
        const float d1z = div255((float)((u1 >> 16) & 0xFFu)), d1w = div255((float)((u1 >> 24) & 0xFFu));
        const f3 pl = F3(frx - (float)ox, fry - (float)oy, frz - (float)oz);
        const float dist = len3(pl);
        const f3 dir = normalize3(pl);
        // the distance along the three directions it faces (the other three would add exact zeros; a NaN
        // direction, at the probe itself, counts as none)
        float hl = sqrt_(mx(fabsf(dir.x), 0.0f)) * (dir.x > 0.0f ? d1x : d1y);
        hl = hl + sqrt_(mx(fabsf(dir.y), 0.0f)) * (dir.y > 0.0f ? d1z : d1w);
        hl = hl + sqrt_(mx(fabsf(dir.z), 0.0f)) * (dir.z > 0.0f ? d0z : d0w);
        if (dist > hl + 0.05f) continue;
        const float wx = ox == 0 ? 1.0f - frx : frx, wy = oy == 0 ? 1.0f - fry : fry, wz = oz == 0 ? 1.0f - frz : frz;
        const float wgt = (wx * wy) * wz;
        res = res + cube_sample_di(cubes + id * 14, n) * wgt;
        tw = tw + wgt;
    }
    if (tw > 0.0f) return F4(div_(res.x, tw), div_(res.y, tw), div_(res.z, tw), div_(res.w, tw));
    return F4(0.0f, 0.0f, 0.0f, 0.0f);
}

// VoxelizeCube (CPUAccelerationStructure.cpp:112-160) for probes [first, first + count).
// VoxelData words: matId, age (0), distances (minDist / unit, inside, +Z, -Z), (+X, -X, +Y, -Y).
__global__ void __launch_bounds__(kVoxThreads) k_probe_voxelize(ShadeScene sc, uint32_t first, uint32_t count,
                                                                uint4* voxels, unsigned long long* counters) {
    __shared__ uint32_t stack[kStackSize * kVoxThreads];
    Counters cn;
    cn.rays = 0; cn.fallbacks = 0; cn.retraces = 0; cn.nodes = 0; cn.tris = 0; cn.hits = 0;
    const uint32_t k = blockIdx.x * kVoxThreads + threadIdx.x;
    if (k < count) {
        const uint32_t g = first + k;
        const f3 o = probe_origin(g);
        uint32_t mat = 0u;
        float dist[6];
#pragma unroll 1
        for (int f = 0; f < 6; ++f) {   // InsideGeometry along +Y, -Y, +X, -X, +Z, -Z
            dist[f] = 255.0f;
            const ProbeHit h = probe_trace(sc, o, face_basis(f), kCubeUnit * 64.0f, stack + threadIdx.x, kVoxThreads, cn);
            if (!h.hit) continue;
            dist[f] = h.t;
            if (h.t <= kCubeUnit) {
                mat = h.mat;
                if (h.back || load_mat(sc, h.mat).model == GKRT_MAT_DIFFUSE_LIGHT) dist[f] = 0.0f;
            }
        }
        float md = mn(mn(mn(mn(mn(dist[0], dist[1]), dist[2]), dist[3]), dist[4]), dist[5]);
        if (md > 254.0f) {
            // DetectDistance along the diagonals (the reference's list repeats two of them)
#pragma unroll 1
            for (int q = 0; q < 6; ++q) {
                const int sx = (q == 0 || q == 3) ? 1 : -1;
                const int sy = (q == 2 || q == 5) ? -1 : 1;
                const int sz = q < 3 ? 1 : -1;
                const f3 d = F3((float)sx * kInvSqrt3, (float)sy * kInvSqrt3, (float)sz * kInvSqrt3);
                const ProbeHit h = probe_trace(sc, o, d, kCubeUnit * 64.0f, stack + threadIdx.x, kVoxThreads, cn);
                md = mn(md, h.hit ? h.t : 255.0f);
            }
        }
        float c[6];
#pragma unroll
        for (int f = 0; f < 6; ++f) c[f] = mn(mx(div_(dist[f], kCubeUnit), 0.0f), 1.0f);
        const float inside = ((((c[0] * c[1]) * c[2]) * c[3]) * c[4]) * c[5];
        const uint32_t w2 = ((uint32_t)div_(md, kCubeUnit) & 0xFFu) | (((uint32_t)(inside * 255.0f) & 0xFFu) << 8) |
                            (((uint32_t)(c[4] * 255.0f) & 0xFFu) << 16) | (((uint32_t)(c[5] * 255.0f) & 0xFFu) << 24);
        const uint32_t w3 = ((uint32_t)(c[2] * 255.0f) & 0xFFu) | (((uint32_t)(c[3] * 255.0f) & 0xFFu) << 8) |
                            (((uint32_t)(c[0] * 255.0f) & 0xFFu) << 16) | (((uint32_t)(c[1] * 255.0f) & 0xFFu) << 24);
        voxels[g] = make_uint4(mat, 0u, w2, w3);
    }
    flush_ray_counters(cn, counters);
}

// ---- the bake ----
struct BakeArgs {
    ProbeLight lt;
    SkySH sh;
    uint32_t first, count;        // probes of this batch
    const uint32_t* cubes_read;   // the grid before the step
    uint32_t* cubes;
    uint4* voxels;
    uint32_t* nlist;              // length of list
    uint32_t* list;               // the batch's surface probes
    float4* light;                // per listed probe, face and face ray: the light it adds
    uint8_t* met;                 // per listed probe, face and ray: it met something
    uint32_t rays;                // rays per face: kFaceRays, light 0, the sun
};

// RenderAmbientCubeOnly bakes surface probes only (a distance byte below 8).
__global__ void __launch_bounds__(256) k_bake_list(BakeArgs a) {
    const uint32_t k = blockIdx.x * 256u + threadIdx.x, lane = threadIdx.x & 31u;
    const bool surface = k < a.count && (a.voxels[a.first + k].z & 0xFFu) < 8u;
    const unsigned m = __ballot_sync(0xFFFFFFFFu, surface);
    uint32_t base = 0;
    if (lane == 0 && m) base = atomicAdd(a.nlist, (uint32_t)__popc(m));
    base = __shfl_sync(0xFFFFFFFFu, base, 0);
    if (surface) a.list[base + __popc(m & ((1u << lane) - 1u))] = a.first + k;
}

struct FaceRay {
    f3 o, d;
    float tmax;
    bool any;
};
// Ray i of face f of probe g: the jittered grid, then light 0, then the sun.
GK_D FaceRay face_ray(const BakeArgs& a, const GkrtFrameConstants& fc, uint32_t g, int f, uint32_t i) {
    const f3 basis = face_basis(f);
    FaceRay r;
    r.o = fma3(basis, kCubeUnit * 0.25f, probe_origin(g));
    r.any = i >= kFaceRays;
    if (!r.any) {
        const uint32_t j = __ldg(&a.voxels[g].y) % 9u;
        const float jx = c_grid3x3[2 * j] * 0.25f, jy = c_grid3x3[2 * j + 1] * 0.25f;
        const f3 hv = normalize3(F3(c_grid4x4[2 * i] + jx, c_grid4x4[2 * i + 1] + jy, 1.0f));
        r.d = align_normal(hv, basis);
        r.tmax = kFastMaxTrace;
    } else if (i == kFaceRays && a.lt.valid) {
        // TraceSegment(origin, lightPos, 0.125): the segment [0.125, len - 0.125] as a ray
        // from origin + 0.125 dir over [EPS, len - 0.25]
        const f3 dv = a.lt.pos - r.o;
        const float len = len3(dv);
        r.d = F3(div_(dv.x, len), div_(dv.y, len), div_(dv.z, len));
        r.o = fma3(r.d, kCubeUnit * 0.5f, r.o);
        r.tmax = len - kCubeUnit;
    } else {
        r.d = F3(fc.sun_direction[0], fc.sun_direction[1], fc.sun_direction[2]);
        r.tmax = kOcclusionMax;
    }
    return r;
}

// The rays of the listed probes as a source of query_run: ray k is ray k mod rays of face
// (k / rays) mod 6 of listed probe k / (6 rays).
struct BakeRays {
    const ShadeScene& sc;
    const GkrtFrameConstants& fc;
    const BakeArgs& a;
    __device__ void split(uint32_t k, uint32_t& p, int& f, uint32_t& i) const {
        p = k / (6u * a.rays);
        const uint32_t r = k - p * 6u * a.rays;
        f = (int)(r / a.rays);
        i = r - (uint32_t)f * a.rays;
    }
    __device__ bool load(uint32_t k, float4& o, float4& d) const {
        uint32_t p, i;
        int f;
        split(k, p, f, i);
        const FaceRay r = face_ray(a, fc, __ldg(&a.list[p]), f, i);
        o = make_float4(r.o.x, r.o.y, r.o.z, kTmin);
        d = make_float4(r.d.x, r.d.y, r.d.z, r.tmax);
        return r.any;
    }
    __device__ void write(const uint4& e, Counters& cn) const {
        uint32_t p, i;
        int f;
        split(e.x, p, f, i);
        const bool hit = e.y != 0xFFFFFFFFu;
        a.met[e.x] = hit ? 1 : 0;
        if (i >= kFaceRays) return;
        const FaceRay r = face_ray(a, fc, __ldg(&a.list[p]), f, i);
        f4 c;
        if (hit) {
            ++cn.hits;
            // the hit material's diffuse times its diffuse texture (AmbientCube.slang:504-510)
            const HitVtx v = hit_vertex(sc, r.o, r.d, e.y, e.z, e.w);
            const MatV m = load_mat(sc, v.mat);
            f4 alb = m.diffuse;
            if (m.dtex >= 0) {
                float tu = 0.0f, tv = 0.0f;   // texture coordinates at the hit (0 without texcoords)
                if (sc.uv) {
                    const HitAttr at = hit_attr(sc, v.i0, v.i1, v.i2, v.b1, v.b2);
                    tu = at.u;
                    tv = at.v;
                }
                alb = alb * tex_sample(sc.tex, m.dtex, tu, tv);
            }
            c = (alb * probe_di(a.cubes_read, sc.voxels, v.P, v.N)) * 1.25f;
        } else {
            c = a.sh.on ? sky_sh(a.sh, fc, r.d) : sky(fc);
        }
        a.light[(size_t)(p * 6u + (uint32_t)f) * kFaceRays + i] = make_float4(c.x, c.y, c.z, c.w);
    }
};

// What bounds it: as the ray queries. Eight lanes per probe, each tracing a face's rays one after
// another, half of the lanes idle beside probes without a surface, took 1.73 ms for a slice of
// 14,720 probes in a field of bricks; the three kernels take 0.52 ms together.
__global__ void __launch_bounds__(kQueryThreads, 4) k_bake_rays(ShadeScene sc, GkrtFrameConstants fc, BakeArgs a, int cap,
                                                               unsigned long long* counters) {
    extern __shared__ __align__(16) uint32_t bake_smem[];
    Counters cn;
    cn.rays = 0; cn.fallbacks = 0; cn.retraces = 0; cn.nodes = 0; cn.tris = 0; cn.hits = 0;
    const BakeRays src{sc, fc, a};
    query_run(sc.S, src, *a.nlist * 6u * a.rays, 32u, cap, bake_smem, cn);
    flush_ray_counters(cn, counters);
}

// The listed probes' new words: 8 lanes per probe, lane f < 6 sums and blends face f.
__global__ void __launch_bounds__(kBakeThreads) k_bake_blend(GkrtFrameConstants fc, BakeArgs a) {
    const uint32_t lane = threadIdx.x & 31u, sub = lane & 7u;
    const uint32_t k = (blockIdx.x * kBakeThreads + threadIdx.x) >> 3;
    const bool valid = k < *a.nlist;
    const uint32_t g = valid ? a.list[k] : 0u;
    const int f = (int)sub;
    uint32_t* cube = a.cubes + (size_t)g * 14u;
    const uint32_t s1 = valid ? cube[13] : 0u;
    // per face: direct word, indirect word, sky-visibility byte (word 12 / 13, byte)
    const int dw = f == 0 ? 8 : f == 1 ? 9 : f == 2 ? 10 : f == 3 ? 11 : f == 4 ? 6 : 7;
    const int iw = dw - 6;
    const int sw = (f == 2 || f == 3) ? 13 : 12;
    const int sb = f == 0 ? 2 : f == 1 ? 3 : f == 2 ? 0 : f == 3 ? 1 : f == 4 ? 0 : 1;
    uint32_t nsky = 0u, nsun = (s1 >> 16) & 0xFFu;
    if (valid && f < 6) {
        const f3 basis = face_basis(f);
        const f3 o = fma3(basis, kCubeUnit * 0.25f, probe_origin(g));
        f4 direct = F4(0.0f, 0.0f, 0.0f, 0.0f), bounce = F4(0.0f, 0.0f, 0.0f, 0.0f);
        float skyv = 0.0f;
        const float4* light = a.light + (size_t)(k * 6u + (uint32_t)f) * kFaceRays;
        const uint8_t* met = a.met + (size_t)(k * 6u + (uint32_t)f) * a.rays;
#pragma unroll 4
        for (uint32_t i = 0; i < kFaceRays; ++i) {
            const float4 c = light[i];
            const f4 c4 = F4(c.x, c.y, c.z, c.w);
            if (met[i]) {
                bounce = bounce + c4;
            } else {
                direct = direct + c4;
                skyv = skyv + 1.0f;
            }
        }
        direct = direct * 0.0625f;
        bounce = bounce * 0.0625f;
        uint32_t next = kFaceRays;
        if (a.lt.valid) {
            const f3 dv = a.lt.pos - o;
            const float len = len3(dv);
            const float atten = met[next++] ? 0.0f : 1.0f;
            const f3 ldir = normalize3(dv);
            const float ndotl = mn(mx(dot3(basis, ldir), 0.0f), 1.0f);
            const float att = div_(ndotl * a.lt.area, (len * len) * 3.14159f);
            direct = direct + (a.lt.power * att) * atten;
        }
        if (fc.has_sun) {
            const f3 sd = F3(fc.sun_direction[0], fc.sun_direction[1], fc.sun_direction[2]);
            const float atten = met[next] ? 0.0f : 1.0f;
            const float ndotl = mn(mx(dot3(basis, sd), 0.0f), 1.0f);
            if (f == 0) nsun = atten > 0.0f ? 1u : 0u;
            const f4 sc4 = F4(fc.sun_color[0], fc.sun_color[1], fc.sun_color[2], fc.sun_color[3]);
            direct = direct + (((sc4 * atten) * ndotl) * 1.0f) * 0.25f;
        }
        const float ov = (float)((cube[sw] >> (8 * sb)) & 0xFFu);
        nsky = (uint32_t)lerpf_(ov, div_(255.0f * skyv, 16.0f), 0.125f) & 0xFFu;
        const f4 od = unpack10(cube[dw]), oi = unpack10(cube[iw]);
        cube[dw] = pack10(F4(lerpf_(od.x, direct.x, 0.125f), lerpf_(od.y, direct.y, 0.125f),
                             lerpf_(od.z, direct.z, 0.125f), lerpf_(od.w, direct.w, 0.125f)));
        cube[iw] = pack10(F4(lerpf_(oi.x, bounce.x, 0.125f), lerpf_(oi.y, bounce.y, 0.125f),
                             lerpf_(oi.z, bounce.z, 0.125f), lerpf_(oi.w, bounce.w, 0.125f)));
    }
    // gather the six sky-visibility bytes (and the sun byte of face +Y) to lane 0 of the group
    const unsigned base = lane & ~7u;
    uint32_t by[6];
#pragma unroll
    for (int q = 0; q < 6; ++q) by[q] = __shfl_sync(0xFFFFFFFFu, nsky, base + q);
    const uint32_t sun = __shfl_sync(0xFFFFFFFFu, nsun, base);
    if (valid && sub == 0u) {
        // word 12: +Z, -Z, +Y, -Y; word 13: +X, -X, sun, unchanged
        cube[12] = by[4] | (by[5] << 8) | (by[0] << 16) | (by[1] << 24);
        cube[13] = by[2] | (by[3] << 8) | ((fc.has_sun ? sun : (s1 >> 16) & 0xFFu) << 16) | (s1 & 0xFF000000u);
        a.voxels[g].y = a.voxels[g].y + 1u;
    }
}

}  // namespace

}  // namespace gk

using namespace gk;

cudaError_t gkrt_launch_probe_voxelize(const ShadeScene& sc, uint32_t first, uint32_t count, uint4* voxels,
                                       unsigned long long* counters, cudaStream_t st) {
    if (count == 0) return cudaSuccess;
    k_probe_voxelize<<<(count + kVoxThreads - 1) / kVoxThreads, kVoxThreads, 0, st>>>(sc, first, count, voxels,
                                                                                     counters);
    return cudaGetLastError();
}

// Probes per batch: 108 MB of scratch at most.
static constexpr uint32_t kBakeBatch = 1u << 16;
bool gkrt_probe_bake_needs_snapshot(uint32_t count) { return count > kBakeBatch; }

cudaError_t gkrt_launch_probe_bake(const ShadeScene& sc, const GkrtFrameConstants& fc, const ProbeLight& lt,
                                   const SkySH& sh, uint32_t first, uint32_t count, const uint32_t* cubes_read,
                                   uint32_t* cubes, uint4* voxels, unsigned long long* counters, int stack_words,
                                   int num_sms, cudaMemPool_t mem, cudaStream_t st) {
    if (count == 0) return cudaSuccess;
    if (stack_words < 1 || stack_words > kQuadStackMax) return cudaErrorInvalidValue;
    static int occ[kMaxDevices][kQuadStackMax + 1] = {};
    const int dev = current_device_slot();
    if (dev < 0) return cudaErrorInvalidDevice;
    int* o = &occ[dev][stack_words];
    const size_t smem = query_smem(stack_words);
    cudaError_t e = cudaSuccess;
    if (!*o) {
        e = cudaFuncSetAttribute(k_bake_rays, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)query_smem(kQuadStackMax));
        if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(o, k_bake_rays, kQueryThreads, smem);
        if (e != cudaSuccess) return e;
    }
    BakeArgs a;
    a.lt = lt;
    a.sh = sh;
    a.cubes_read = cubes_read;
    a.cubes = cubes;
    a.voxels = voxels;
    a.rays = kFaceRays + (lt.valid ? 1u : 0u) + (fc.has_sun ? 1u : 0u);
    // scratch of this call alone: light, list and its length, flags
    const uint32_t batch = std::min(count, kBakeBatch);
    const size_t nlight = (size_t)batch * 6u * kFaceRays, nmet = (size_t)batch * 6u * a.rays;
    uint8_t* p = nullptr;
    e = cudaMallocFromPoolAsync((void**)&p, nlight * sizeof(float4) + 16u + (size_t)batch * 4u + nmet, mem, st);
    if (e != cudaSuccess) return e;
    a.light = reinterpret_cast<float4*>(p);
    a.nlist = reinterpret_cast<uint32_t*>(p + nlight * sizeof(float4));
    a.list = a.nlist + 4;
    a.met = reinterpret_cast<uint8_t*>(a.list + batch);
    const uint32_t most = (uint32_t)(num_sms * std::max(1, *o));
    for (uint32_t at = 0; at < count && e == cudaSuccess; at += batch) {
        a.first = first + at;
        a.count = std::min(batch, count - at);
        e = cudaMemsetAsync(a.nlist, 0, 4, st);
        if (e != cudaSuccess) break;
        k_bake_list<<<(a.count + 255u) / 256u, 256, 0, st>>>(a);
        const uint32_t need = (uint32_t)(((uint64_t)a.count * 6u * a.rays + 32u * kQueryWarps - 1u) / (32u * kQueryWarps));
        k_bake_rays<<<std::min(most, need), kQueryThreads, smem, st>>>(sc, fc, a, stack_words, counters);
        k_bake_blend<<<(a.count * 8u + kBakeThreads - 1u) / kBakeThreads, kBakeThreads, 0, st>>>(fc, a);
        e = cudaGetLastError();
    }
    const cudaError_t ef = cudaFreeAsync(p, st);
    return e == cudaSuccess ? ef : e;
}
