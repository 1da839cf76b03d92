// gk_trace.cuh — two-level BVH traversal with an exact closest-hit contract (sm_103a).
//
// Replaces the RT-core RayQuery of FHardwareRayTracerV2 (assets/shaders/common/
// Shading.slang:737-826). GB300 has no RT cores, so traversal is software, over either of
// the two node formats the builders produce from the same SAH trees:
//   * four-child nodes (128 bytes, one cache line, seven 16-byte loads per node, a stack of
//     node refs): used by the rt pass, the adjoint, the ray queries and the probe bake;
//   * compressed 8-wide nodes (96 bytes, six loads test eight 8-bit child boxes, a stack of
//     sorted node groups): used by the probe voxelization.
// Both keep 48-byte triangles in leaf order, a per-thread stack in shared memory (strided
// by the block size, conflict-free) and a marker entry for the hand-over from the instance
// level to the mesh level.
//
// Hit contract. The reported hit is the minimum of (t, instance index, primitive index)
// under an FP64 evaluation of the watertight ray/triangle test (Woop, Benthin, Wald,
// JCGT 2013) on the FP32 object-space ray. The kernel computes in FP32 with certified
// error bounds and uses FP64 only where the bounds do not decide:
//   * edge functions U, V, W within their error bound of zero -> FP64 test;
//   * t within its error bound of tmin/tmax -> FP64 t;
//   * two hits whose t-intervals overlap -> both are decided in FP64 (the incumbent's
//     triangle is fetched again) and the key is compared exactly.
// Box tests widen the slab interval by 1e-6 relative (> 2.5 gamma_3; quad_slabs adds what its
// fused form needs), so no box holding the FP64 winner is culled. A ray component of exactly zero lying on a box face is the one
// case a t-interval widening cannot cover ((hi - o) * inv is 0 there), so the builders store
// every node box widened in space as well (widen_lo / widen_hi): a triangle edge on the
// face stays inside the box the ray is tested against. The 8-bit child boxes of the wide
// nodes decode EXACTLY to planes at or outside those widened boxes (WideNode below), so the
// compression adds boxes, never removes them. The float t and barycentrics used for shading
// are those of the FP32 test when it is certain, else the rounded FP64 values.
#pragma once
#include "gk_device.cuh"

namespace gk {

// Two-child node: the output of the SAH builders, collapsed into QuadNode and WideNode for
// traversal.
struct __align__(16) BvhNode {
    float4 a;   // c0.lo.x c0.lo.y c0.lo.z c0.hi.x
    float4 b;   // c0.hi.y c0.hi.z c1.lo.x c1.lo.y
    float4 c;   // c1.lo.z c1.hi.x c1.hi.y c1.hi.z
    int4 d;     // ref0 ref1 - -   (ref >= 0: interior node; ref < 0: ~(payload << 3 | count-1))
};

// Four-child node: the quad of two-child node n is quad n, so that a collapse needs no
// compaction and a refit rewrites quads in place (half of the slots are never visited). Its
// children are n's grandchildren, a leaf child of n staying as it is (and its place taken by a
// child of the largest interior grandchild), so every interior child lies at least two levels
// below n and a ray needs at most 3 stack entries per two levels. Planes are stored per axis and
// side for the four children, so that a ray loads its near and far planes by the sign of its
// direction instead of ordering them. A slot without a child has ref kRefPop and a box that no
// finite ray meets; popping it pops again.
struct __align__(16) QuadNode {
    float4 p[6];    // lo.x hi.x lo.y hi.y lo.z hi.z, child j in component j
    int4 ref;       // BvhNode encoding
    int4 pad;       // one node per 128-byte line
};

// Compressed 8-wide node. Per axis a scale s = 2^e (-100 <= e <= 38) and an integer origin k
// (|k| < 2^22, origin p = k s exact in float); child slot j's planes are (k + q) s for 8-bit
// q_lo = floor(lo / s) - 1 - k and q_hi = ceil(hi / s) + 1 - k of the child's stored (widened)
// box: every encoded box lies at least one step s outside the box it encodes.
// Traversal evaluates a plane's t as fma(2^23 + q, C, B') with C = s inv (exact) and
// B' = (p - o) inv - 2^23 C (three roundings), whose error is below 5.02u|t| + 0.5001 s|inv|:
// the step margin absorbs the absolute part and the 1e-6 slab widening the relative part, so
// no box holding the exact winner is culled.
struct __align__(16) WideNode {
    float4 h;       // origin p x y z; w bits: 0-7 / 8-15 / 16-23 = e + 127 per axis, 24-31 valid-slot mask
    uint4 q[3];     // per axis: q_lo slots 0-3, q_lo 4-7, q_hi 0-3, q_hi 4-7 (slot j in byte j & 3)
    int4 ref[2];    // slot refs, BvhNode encoding (interior refs index the WideNode array)
};

struct __align__(16) DevInst {
    float winv[12];       // world -> object rows
    int blas_root;        // root node index of the mesh BVH
    uint32_t index_offset;
    uint32_t vertex_offset;
    uint32_t instance_id;
    int blas_wide_root;   // root WideNode index of the mesh BVH
    uint32_t pad[3];
};

// Node boxes as stored: 1e-6 relative plus 1e-10 absolute beyond the primitives' bounds.
GK_HD float widen_lo(float v) { return v - (fabsf(v) * 1e-6f + 1e-10f); }
GK_HD float widen_hi(float v) { return v + (fabsf(v) * 1e-6f + 1e-10f); }

constexpr int kStackEntries = 24;                // wide node-group entries per thread (3 words each)
constexpr int kStackSize = 3 * kStackEntries;    // 32-bit words per thread
constexpr int kMaxBinLevels = kStackSize - 3;    // two-child levels of both trees a build may have
// Stack words of a ray over quad nodes for trees of the given two-child depths (root = 0): three
// refs per two levels of each tree, and the marker.
GK_HD constexpr int quad_stack_words(int blas_depth, int tlas_depth) {
    return 3 * (blas_depth / 2 + 1) + 3 * (tlas_depth / 2 + 1) + 1;
}
constexpr int kQuadStackMax = 3 * (kMaxBinLevels / 2 + 2) + 1;
constexpr int kRefPop = 0x7FFFFFFE;
constexpr int kRefMarker = 0x7FFFFFFF;
constexpr int kIterCap = 1 << 22;
// Speculative traversal (keep taking node steps while a found leaf waits for the leaf phase)
// is measured slower here: a lane stops at its first leaf.
constexpr bool kSpeculative = false;   // measured: 4.01 ms without, 4.16 ms with (1080p bricks)
constexpr uint32_t kErrStack = 1u, kErrIter = 2u;
// (4u is the TMA wait timeout of the post passes, gk_tma.cuh)
constexpr uint32_t kErrRefit = 8u;   // a refit box that the 8-wide nodes cannot quantize
constexpr uint32_t kErrBounds = 16u;  // checked builds: an index outside its array (access skipped)

// Checked builds (GKRT_CHECKED) test every node, triangle and instance index against its array
// before the access; a bad index records kErrBounds, ends the ray and skips the access. The
// default build compiles the checks away.
#ifdef GKRT_CHECKED
#define GK_CHECK_OR_END(ok, S, T, ret)              \
    do {                                            \
        if (!(ok)) {                                \
            atomicOr((S).error, kErrBounds);        \
            (T).done = true;                        \
            (T).has_leaf = false;                   \
            return ret;                             \
        }                                           \
    } while (0)
#else
#define GK_CHECK_OR_END(ok, S, T, ret) \
    do {                               \
    } while (0)
#endif

// Per-thread event counts, flushed once per warp at the end of a kernel. Context counter
// slots: 0 rays, 1 FP64 fallbacks, 2 exact re-traces, 3 node visits, 4 triangle tests,
// 5 hit fetches (closest hits whose vertex, normal, material and instance data were read),
// all per pass; 6 rays since the context was created.
struct Counters {
    uint32_t rays, fallbacks, retraces, nodes, tris, hits;
};

struct SceneView {
    const float4* quad;     // QuadNode array
    const WideNode* wide;   // the same trees collapsed into 8-wide nodes
    const float4* tris;     // 3 float4 per triangle, v0.w = primitive index bits
    const DevInst* inst;
    int tlas_root;          // quad root of the instance level, -1: empty scene
    int tlas_wide_root;     // wide root of the instance level
    uint32_t* error;
    uint32_t node_count, wide_count, tri_count, inst_count;   // array sizes (checked builds)
};

struct Shear {
    int kx, ky, kz;
    float Sx, Sy, Sz;
};

GK_D float rcp_approx(float x) {
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}
GK_D float max3f(float a, float b, float c) { return fmaxf(fmaxf(a, b), c); }
GK_D float min3f(float a, float b, float c) { return fminf(fminf(a, b), c); }

GK_D float pick(f3 v, int k) { return k == 0 ? v.x : (k == 1 ? v.y : v.z); }

GK_D Shear make_shear(f3 d) {
    Shear s;
    float ax = fabsf(d.x), ay = fabsf(d.y), az = fabsf(d.z);
    int kz = 0;
    float am = ax;
    if (ay > am) { kz = 1; am = ay; }
    if (az > am) { kz = 2; }
    int kx = kz == 2 ? 0 : kz + 1;
    int ky = kx == 2 ? 0 : kx + 1;
    float dz = pick(d, kz);
    if (dz < 0.0f) { int t = kx; kx = ky; ky = t; }
    float dx = pick(d, kx), dy = pick(d, ky);
    s.kx = kx; s.ky = ky; s.kz = kz;
    s.Sx = div_(dx, dz);
    s.Sy = div_(dy, dz);
    s.Sz = rcp_(dz);
    return s;
}

// FP64 shear constants, computed only when an FP64 decision is needed.
struct ShearD { double Sxd, Syd, Szd; };
GK_D ShearD shear_d(f3 d, const Shear& s) {
    const double dz = (double)pick(d, s.kz);
    ShearD r;
    r.Sxd = (double)pick(d, s.kx) / dz;
    r.Syd = (double)pick(d, s.ky) / dz;
    r.Szd = 1.0 / dz;
    return r;
}

struct ExactHit { bool hit; double t, b1, b2; };

// FP64 watertight test; products and sums rounded in double, nothing fused.
// Out of line, shear included: taken rarely, and inlining it at every call site bloats the hot
// kernels.
static __device__ __noinline__ ExactHit exact_test(f3 o, f3 d, f3 v0, f3 v1, f3 v2) {
    ExactHit r; r.hit = false; r.t = 0.0; r.b1 = 0.0; r.b2 = 0.0;
    const Shear s = make_shear(d);
    const ShearD sd = shear_d(d, s);
    double Ak = (double)pick(v0, s.kz) - (double)pick(o, s.kz);
    double Bk = (double)pick(v1, s.kz) - (double)pick(o, s.kz);
    double Ck = (double)pick(v2, s.kz) - (double)pick(o, s.kz);
    double Ax = ((double)pick(v0, s.kx) - (double)pick(o, s.kx)) - sd.Sxd * Ak;
    double Ay = ((double)pick(v0, s.ky) - (double)pick(o, s.ky)) - sd.Syd * Ak;
    double Bx = ((double)pick(v1, s.kx) - (double)pick(o, s.kx)) - sd.Sxd * Bk;
    double By = ((double)pick(v1, s.ky) - (double)pick(o, s.ky)) - sd.Syd * Bk;
    double Cx = ((double)pick(v2, s.kx) - (double)pick(o, s.kx)) - sd.Sxd * Ck;
    double Cy = ((double)pick(v2, s.ky) - (double)pick(o, s.ky)) - sd.Syd * Ck;
    double U = Cx * By - Cy * Bx;
    double V = Ax * Cy - Ay * Cx;
    double W = Bx * Ay - By * Ax;
    bool in = (U >= 0.0 && V >= 0.0 && W >= 0.0) || (U <= 0.0 && V <= 0.0 && W <= 0.0);
    if (!in) return r;
    double det = U + V + W;
    if (det == 0.0) return r;
    double T = U * (sd.Szd * Ak) + V * (sd.Szd * Bk) + W * (sd.Szd * Ck);
    r.hit = true;
    r.t = T / det;
    r.b1 = V / det;
    r.b2 = W / det;
    return r;
}

struct Fp32Hit { int kind; float t, b1, b2; };   // kind: 0 certain miss, 1 certain hit, 2 undecided

// FP32 test with certified bounds on U, V, W (first order: 3.02u x magnitude x lateral
// offset), for the shading values of a hit. Unit roundoff u = 2^-24.
GK_D Fp32Hit fp32_test(f3 o, const Shear& s, f3 v0, f3 v1, f3 v2) {
    const float kU = 5.9604645e-08f;
    Fp32Hit r; r.kind = 0; r.t = 0.0f; r.b1 = 0.0f; r.b2 = 0.0f;
    f3 a = v0 - o, b = v1 - o, c = v2 - o;
    float akx = pick(a, s.kx), aky = pick(a, s.ky), akz = pick(a, s.kz);
    float bkx = pick(b, s.kx), bky = pick(b, s.ky), bkz = pick(b, s.kz);
    float ckx = pick(c, s.kx), cky = pick(c, s.ky), ckz = pick(c, s.kz);
    float Ax = fmaf_(-s.Sx, akz, akx), Ay = fmaf_(-s.Sy, akz, aky);
    float Bx = fmaf_(-s.Sx, bkz, bkx), By = fmaf_(-s.Sy, bkz, bky);
    float Cx = fmaf_(-s.Sx, ckz, ckx), Cy = fmaf_(-s.Sy, ckz, cky);
    float U = fmaf_(Cx, By, -(Cy * Bx));
    float V = fmaf_(Ax, Cy, -(Ay * Cx));
    float W = fmaf_(Bx, Ay, -(By * Ax));
    float aSx = fabsf(s.Sx), aSy = fabsf(s.Sy);
    float mAx = fmaf_(aSx, fabsf(akz), fabsf(akx)), mAy = fmaf_(aSy, fabsf(akz), fabsf(aky));
    float mBx = fmaf_(aSx, fabsf(bkz), fabsf(bkx)), mBy = fmaf_(aSy, fabsf(bkz), fabsf(bky));
    float mCx = fmaf_(aSx, fabsf(ckz), fabsf(ckx)), mCy = fmaf_(aSy, fabsf(ckz), fabsf(cky));
    // first-order error: magnitude x lateral offset (3.02u), second order 9.2u^2 magnitude^2,
    // product/result rounding u|Cy Bx| + 1.01u|U|; constants rounded up to 4u, 16u^2, 2u
    const float kA = 4.0f * kU, kB = 2.0f * kU, kC = 16.0f * kU * kU;
    float eU = fmaf_(kA, fmaf_(mCx, fabsf(By), fmaf_(fabsf(Cx), mBy, fmaf_(mCy, fabsf(Bx), fabsf(Cy) * mBx))),
                     fmaf_(kC, fmaf_(mCx, mBy, mCy * mBx), kB * (fabsf(Cy * Bx) + fabsf(U))));
    float eV = fmaf_(kA, fmaf_(mAx, fabsf(Cy), fmaf_(fabsf(Ax), mCy, fmaf_(mAy, fabsf(Cx), fabsf(Ay) * mCx))),
                     fmaf_(kC, fmaf_(mAx, mCy, mAy * mCx), kB * (fabsf(Ay * Cx) + fabsf(V))));
    float eW = fmaf_(kA, fmaf_(mBx, fabsf(Ay), fmaf_(fabsf(Bx), mAy, fmaf_(mBy, fabsf(Ax), fabsf(By) * mAx))),
                     fmaf_(kC, fmaf_(mBx, mAy, mBy * mAx), kB * (fabsf(By * Ax) + fabsf(W))));
    bool pos = (U > eU) || (V > eV) || (W > eW);
    bool ng = (U < -eU) || (V < -eV) || (W < -eW);
    if (pos && ng) return r;
    bool allpos = (U > eU) && (V > eV) && (W > eW);
    bool allneg = (U < -eU) && (V < -eV) && (W < -eW);
    if (!(allpos || allneg)) { r.kind = 2; return r; }
    float det = (U + V) + W;
    float adet = fabsf(det);
    float ED = fmaf_(2.01f * kU, adet, (eU + eV) + eW);
    if (ED >= 0.5f * adet) { r.kind = 2; return r; }
    float Az = s.Sz * akz, Bz = s.Sz * bkz, Cz = s.Sz * ckz;
    float T = fmaf_(W, Cz, fmaf_(V, Bz, U * Az));
    r.kind = 1;
    r.t = div_(T, det);
    r.b1 = div_(V, det);
    r.b2 = div_(W, det);
    return r;
}

// The traversal's ray / triangle test: which side of certain the FP64 test's answer lies, and a
// certified interval [t - e, t + e] of its distance. Only this classification and the FP64
// fallback decide hits, so any formula with a certified bound serves; the edge form (Moeller and
// Trumbore 1997) needs no shear and no axis permutation, and its scalar triple products give the
// distance as well. With w = o - v0, e1 = v1 - v0, e2 = v2 - v0, p = d x e2, q = w x e1:
//   u = w . p, v = d . q, x = det - u - v (the three edges), det = e1 . p, t = (e2 . q) / det.
// Errors, in units of u = 2^-24 times the sum of the absolute products: the differences carry 1
// each, a cross product's component 3 (p) or 4 (q) with them, a dot product 3 more: det, u and v
// 7, e2 . q 8; the constants below are rounded up for the second order and the sums' own
// rounding (and 1e-37 covers products that underflow). x adds the three errors and 2 roundings. As in the FP32 shading test, edges that are
// not certain, or errors above half of det, leave the decision to FP64. The reciprocals are
// approximate (2 ulps, inside the slack of 1.25 and 8u |t|) and flushed to zero for a determinant above
// 2^126, which is left to FP64 too. The last term covers the FP64
// test's own error: 2^-29 of an FP32 evaluation's, itself below the farthest vertex's distance.
struct TriTest { int kind; float t, e; };   // kind: 0 certain miss, 1 certain hit, 2 undecided
GK_D TriTest tri_test(f3 o, f3 d, f3 v0, f3 v1, f3 v2) {
    const float kU = 5.9604645e-08f;
    TriTest r; r.kind = 0; r.t = 0.0f; r.e = 0.0f;
    const f3 w = o - v0, e1 = v1 - v0, e2 = v2 - v0;
    const float p0 = d.z * e2.y, p1 = d.x * e2.z, p2 = d.y * e2.x;
    const f3 p = F3(fmaf_(d.y, e2.z, -p0), fmaf_(d.z, e2.x, -p1), fmaf_(d.x, e2.y, -p2));
    const f3 A = F3(fmaf_(fabsf(d.y), fabsf(e2.z), fabsf(p0)), fmaf_(fabsf(d.z), fabsf(e2.x), fabsf(p1)),
                    fmaf_(fabsf(d.x), fabsf(e2.y), fabsf(p2)));
    const float q0 = w.z * e1.y, q1 = w.x * e1.z, q2 = w.y * e1.x;
    const f3 q = F3(fmaf_(w.y, e1.z, -q0), fmaf_(w.z, e1.x, -q1), fmaf_(w.x, e1.y, -q2));
    const f3 B = F3(fmaf_(fabsf(w.y), fabsf(e1.z), fabsf(q0)), fmaf_(fabsf(w.z), fabsf(e1.x), fabsf(q1)),
                    fmaf_(fabsf(w.x), fabsf(e1.y), fabsf(q2)));
    const float det = dot3(e1, p), u = dot3(w, p), v = dot3(d, q);
    const float x = (det - u) - v;
    const float sd = fmaf_(fabsf(e1.z), A.z, fmaf_(fabsf(e1.y), A.y, fabsf(e1.x) * A.x));
    const float su = fmaf_(fabsf(w.z), A.z, fmaf_(fabsf(w.y), A.y, fabsf(w.x) * A.x));
    const float sv = fmaf_(fabsf(d.z), B.z, fmaf_(fabsf(d.y), B.y, fabsf(d.x) * B.x));
    const float eu = fmaf_(8.0f * kU, su, 1e-37f), ev = fmaf_(8.0f * kU, sv, 1e-37f),
                ex = fmaf_(11.0f * kU, (sd + su) + sv, 1e-37f);
    const bool pos = (u > eu) || (v > ev) || (x > ex);
    const bool ng = (u < -eu) || (v < -ev) || (x < -ex);
    if (pos && ng) return r;
    const bool allpos = (u > eu) && (v > ev) && (x > ex);
    const bool allneg = (u < -eu) && (v < -ev) && (x < -ex);
    const float adet = fabsf(det);
    r.kind = 2;
    if (!(allpos || allneg) || !(ex < 0.5f * adet) || !(adet < 0x1p126f)) return r;
    const float ed = (8.0f * kU) * sd;
    const float t = dot3(e2, q) * rcp_approx(det);
    const float et = (10.0f * kU) * fmaf_(fabsf(e2.z), B.z, fmaf_(fabsf(e2.y), B.y, fabsf(e2.x) * B.x));
    const float at = fabsf(t);
    const float far = (max3f(fabsf(w.x), fabsf(w.y), fabsf(w.z)) +
                       fmaxf(max3f(fabsf(e1.x), fabsf(e1.y), fabsf(e1.z)), max3f(fabsf(e2.x), fabsf(e2.y), fabsf(e2.z)))) *
                      rcp_approx(max3f(fabsf(d.x), fabsf(d.y), fabsf(d.z)));
    r.kind = 1;
    r.t = t;
    r.e = fmaf_(1.25f * fmaf_(at, ed, et), rcp_approx(adet - ed), fmaf_(8.0f * kU, at, 3e-8f * far));
    return r;
}

GK_D f3 safe_inv(f3 d) {
    float x = fabsf(d.x) < 1e-20f ? copysignf(1e-20f, d.x) : d.x;
    float y = fabsf(d.y) < 1e-20f ? copysignf(1e-20f, d.y) : d.y;
    float z = fabsf(d.z) < 1e-20f ? copysignf(1e-20f, d.z) : d.z;
    return F3(rcp_(x), rcp_(y), rcp_(z));
}

// Slab constants of a ray over quad nodes. A plane p is met at t = (p - o) inv, evaluated as one
// fused multiply-add, near t = fma(p, inv, nn) and far t = fma(p, inv, nf) with nn, nf = -o inv
// shifted by 4u |o inv|: the product's rounding and the shift's own are at most 2u |o inv|, so nn
// is at or below -o inv and nf at or above it by what those roundings can cost, and the fused
// step's u |t| and the reciprocal's error (2 ulps, a common factor of the three terms) are covered
// by the 1e-6 relative widening. inv: an approximate reciprocal suffices, |d| at least 1e-20.
struct Slabs {
    f3 inv, nn, nf;
};
GK_D void slab_axis(float o, float d, float& inv, float& nn, float& nf) {
    inv = rcp_approx(fabsf(d) < 1e-20f ? copysignf(1e-20f, d) : d);
    const float oi = o * inv, m = fabsf(oi) * 2.3841858e-07f;   // 4u
    nn = -oi - m;
    nf = -oi + m;
}
GK_D Slabs quad_slabs(f3 o, f3 d) {
    Slabs s;
    slab_axis(o.x, d.x, s.inv.x, s.nn.x, s.nf.x);
    slab_axis(o.y, d.y, s.inv.y, s.nn.y, s.nf.y);
    slab_axis(o.z, d.z, s.inv.z, s.nn.z, s.nf.z);
    return s;
}

// tnear of one child's box over [tmin, tcull] (widened by 1e-6 relative, as tcull is), +inf when
// the ray misses it.
GK_D float quad_near(float nx, float ny, float nz, float fx, float fy, float fz, const Slabs& s, float tmin,
                     float tcull) {
    const float tn = fmaxf(max3f(fmaf_(nx, s.inv.x, s.nn.x), fmaf_(ny, s.inv.y, s.nn.y), fmaf_(nz, s.inv.z, s.nn.z)),
                           tmin);
    const float tf = min3f(fmaf_(fx, s.inv.x, s.nf.x), fmaf_(fy, s.inv.y, s.nf.y), fmaf_(fz, s.inv.z, s.nf.z)) *
                     1.000001f;
    return tn <= fminf(tf, tcull) ? tn : __int_as_float(0x7F800000);
}

// Orders two children by tnear.
GK_D void quad_cx(float& ta, int& ra, float& tb, int& rb) {
    const bool s = tb < ta;
    const float t = s ? tb : ta;
    tb = s ? ta : tb;
    ta = t;
    const int r = s ? rb : ra;
    rb = s ? ra : rb;
    ra = r;
}

struct TraceOut {
    bool hit;
    bool ambiguous;
    uint32_t inst, prim, tri;
};

enum { kClosest = 0, kAny = 1 };

// The world -> object rows of an instance, three 16-byte loads.
GK_D void load_winv(const DevInst* ip, float (&w)[12]) {
    const float4* p = reinterpret_cast<const float4*>(ip->winv);
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const float4 v = __ldg(p + k);
        w[4 * k] = v.x; w[4 * k + 1] = v.y; w[4 * k + 2] = v.z; w[4 * k + 3] = v.w;
    }
}

GK_D f3 tri_v(const float4* tris, uint32_t ti, int k, uint32_t* prim = nullptr) {
    float4 v = __ldg(&tris[3 * ti + k]);
    if (prim) *prim = __float_as_uint(v.w);
    return F3(v.x, v.y, v.z);
}

// Resumable traversal state of one ray. The stack lives in shared memory (caller-owned,
// strided); everything else is here, so a ray can be advanced one step at a time and a
// lane can leave the traversal loop and come back.
struct Trav {
    f3 wo, wd;            // world ray (restored on leaving an instance)
    f3 o, d;              // ray in the current space (world or instance)
    Slabs sl;             // its slab constants (quad nodes)
    f3 inv;               // its safe reciprocal direction (8-wide nodes)
    float tmin;           // read by the ray-query kernels (kRayTmin); the rt pass uses kTmin
    float tmax, tcull, best_lo, best_hi;
    double best_td;
    uint32_t inst, prim, tri;   // current best
    uint32_t cur;               // instance being traversed
    int ref, sp, iter;
    int mode;                   // kClosest / kAny
    uint32_t leaf;              // postponed triangle leaf (payload), valid when has_leaf
    bool hit, best_exact, inblas, done, ambiguous, has_leaf;
};

constexpr float kTmin = 1e-3f;   // EPS, assets/shaders/common/PreProcessor.slang:13

// tmin: the ray's lower bound, honoured by the functions instantiated with kRayTmin (the ray
// queries); the rt pass and the bake kernels trace every ray from EPS and keep it a constant.
template <bool kWide = false>
GK_D void trav_init(Trav& T, const SceneView& S, f3 wo, f3 wd, float tmax, int mode, float tmin = kTmin) {
    T.wo = wo; T.wd = wd; T.o = wo; T.d = wd;
    if (kWide) T.inv = safe_inv(wd);
    else T.sl = quad_slabs(wo, wd);
    T.tmin = tmin;
    T.tmax = tmax;
    T.tcull = tmax * 1.000001f;
    T.best_lo = 0.0f; T.best_hi = 0.0f; T.best_td = 0.0;
    T.inst = 0xFFFFFFFFu; T.prim = 0xFFFFFFFFu; T.tri = 0xFFFFFFFFu;
    T.cur = 0; T.sp = 0; T.iter = 0;
    T.mode = mode;
    T.hit = false; T.best_exact = false; T.inblas = false; T.ambiguous = false;
    T.has_leaf = false; T.leaf = 0u;
    T.ref = kWide ? S.tlas_wide_root : S.tlas_root;
    T.done = T.ref < 0;
}

// FP64 t of the current best candidate: its triangle against its instance's
// object-space ray (recomputed with the same FP32 operations as during traversal).
GK_D double exact_t_of(const Trav& T, const SceneView& S) {
    f3 o = T.o, d = T.d;
    if (!T.inblas || T.inst != T.cur) {
        float w[12];
        load_winv(S.inst + T.inst, w);
        o = xpoint(w, T.wo);
        d = xvector(w, T.wd);
    }
    return exact_test(o, d, tri_v(S.tris, T.tri, 0), tri_v(S.tris, T.tri, 1), tri_v(S.tris, T.tri, 2)).t;
}

// Test the triangles of one leaf against the current best. Returns true when the ray is
// finished early (any-hit found). kRayTmin: the ray's own tmin, else the constant EPS.
template <bool kRayTmin = false>
GK_D bool trav_leaf(Trav& T, const SceneView& S, uint32_t first, uint32_t cnt, Counters& cn) {
    const float tmin = kRayTmin ? T.tmin : kTmin;
    const double tmind = (double)tmin, tmaxd = (double)T.tmax;
    for (uint32_t k = 0; k < cnt; ++k) {
        const uint32_t ti = first + k;
        uint32_t prim;
        const f3 v0 = tri_v(S.tris, ti, 0, &prim), v1 = tri_v(S.tris, ti, 1), v2 = tri_v(S.tris, ti, 2);
        ++cn.tris;
        const TriTest f = tri_test(T.o, T.d, v0, v1, v2);
        if (f.kind == 0) continue;
        float t = f.t, e = f.e;
        double td = 0.0;
        bool have_td = false;
        if (f.kind == 2) {
            const ExactHit x = exact_test(T.o, T.d, v0, v1, v2);
            ++cn.fallbacks;
            if (!x.hit) continue;
            td = x.t; have_td = true;
            t = (float)x.t;
            e = 2.384185791e-07f * fabsf(t);   // 4u |t|
        }
        if (t + e < tmin || t - e > T.tmax) continue;
        if (t - e < tmin || t + e > T.tmax) {
            if (!have_td) {
                const ExactHit x = exact_test(T.o, T.d, v0, v1, v2);
                ++cn.fallbacks;
                td = x.t; have_td = true;
                t = (float)x.t;
                e = 2.384185791e-07f * fabsf(t);
            }
            if (!(td >= tmind && td <= tmaxd)) continue;
        }
        if (T.mode == kAny) {
            T.hit = true; T.inst = T.cur; T.prim = prim; T.tri = ti;
            return true;
        }
        const float lo = t - e, hi = t + e;
        if (T.hit) {
            if (have_td && T.best_exact) {
                // both FP64: compare the key (t, instance, primitive) exactly
                const bool closer = td < T.best_td ||
                                    (td == T.best_td && (T.cur < T.inst || (T.cur == T.inst && prim < T.prim)));
                if (!closer) continue;
            } else {
                if (lo > T.best_hi) continue;
                if (!(hi < T.best_lo)) {
                    // intervals overlap: decide both in FP64 and compare the key exactly
                    ++cn.retraces;
                    if (!have_td) {
                        const ExactHit x = exact_test(T.o, T.d, v0, v1, v2);
                        ++cn.fallbacks;
                        td = x.t; have_td = true;
                        t = (float)x.t;
                        e = 2.384185791e-07f * fabsf(t);
                    }
                    if (!T.best_exact) {
                        T.best_td = exact_t_of(T, S);
                        T.best_exact = true;
                        ++cn.fallbacks;
                    }
                    const bool closer = td < T.best_td ||
                                        (td == T.best_td && (T.cur < T.inst || (T.cur == T.inst && prim < T.prim)));
                    if (!closer) continue;
                }
            }
        }
        T.hit = true; T.inst = T.cur; T.prim = prim; T.tri = ti;
        T.best_lo = lo; T.best_hi = hi;
        T.best_exact = have_td;
        T.best_td = td;
        T.tcull = hi * 1.000001f;
    }
    return false;
}

// ---- traversal over quad nodes ----
// A ray is always in one of four states, so that a warp can run one kind of work at a time for
// all the lanes that need it: kStNode (T.ref is an interior node to test), kStTrans (an instance
// to enter, or the marker: the instance just traversed to leave), kStLeaf (a triangle leaf to
// test) and kStDone.
enum TravState : int { kStDone = 0, kStNode = 1, kStTrans = 2, kStLeaf = 3 };

// The next reference to visit, `ref` or the top of the stack, and the state it puts the ray in.
GK_D int trav_next(Trav& T, int ref, const uint32_t* stk, int stride) {
    while (ref == kRefPop) {
        if (T.sp == 0) return kStDone;
        --T.sp;
        ref = (int)stk[T.sp * stride];
    }
    T.ref = ref;
    return ref == kRefMarker ? kStTrans : ref >= 0 ? kStNode : T.inblas ? kStLeaf : kStTrans;
}

// Tests the four children of node T.ref: the nearest met is visited next, the others are pushed,
// farthest first. cap: the stack's capacity in words; the caller's stack holds cap * stride.
// kRayTmin: the ray's own tmin, else the constant EPS.
template <bool kRayTmin = false>
GK_D int trav_node(Trav& T, const SceneView& S, uint32_t* stk, int stride, Counters& cn, int cap) {
    if (++T.iter > kIterCap) { atomicOr(S.error, kErrIter); return kStDone; }
    GK_CHECK_OR_END((uint32_t)T.ref < S.node_count, S, T, kStDone);
    ++cn.nodes;
    const float tmin = kRayTmin ? T.tmin : kTmin;
    // plane rows by the direction's signs: near lo and far hi for a positive component
    const uint32_t row = 8u * (uint32_t)T.ref;
    const uint32_t ix = row | (__float_as_uint(T.sl.inv.x) >> 31), iy = row | 2u | (__float_as_uint(T.sl.inv.y) >> 31),
                   iz = row | 4u | (__float_as_uint(T.sl.inv.z) >> 31);
    const float4 nx = __ldg(S.quad + ix), fx = __ldg(S.quad + (ix ^ 1u));
    const float4 ny = __ldg(S.quad + iy), fy = __ldg(S.quad + (iy ^ 1u));
    const float4 nz = __ldg(S.quad + iz), fz = __ldg(S.quad + (iz ^ 1u));
    const int4 rf = __ldg(reinterpret_cast<const int4*>(S.quad + (row | 6u)));
    float t0 = quad_near(nx.x, ny.x, nz.x, fx.x, fy.x, fz.x, T.sl, tmin, T.tcull);
    float t1 = quad_near(nx.y, ny.y, nz.y, fx.y, fy.y, fz.y, T.sl, tmin, T.tcull);
    float t2 = quad_near(nx.z, ny.z, nz.z, fx.z, fy.z, fz.z, T.sl, tmin, T.tcull);
    float t3 = quad_near(nx.w, ny.w, nz.w, fx.w, fy.w, fz.w, T.sl, tmin, T.tcull);
    int r0 = rf.x, r1 = rf.y, r2 = rf.z, r3 = rf.w;
    quad_cx(t0, r0, t1, r1); quad_cx(t2, r2, t3, r3); quad_cx(t0, r0, t2, r2); quad_cx(t1, r1, t3, r3);
    quad_cx(t1, r1, t2, r2);
    const float inf = __int_as_float(0x7F800000);
    const int more = t3 < inf ? 3 : t2 < inf ? 2 : t1 < inf ? 1 : 0;
    if (T.sp + more > cap) { atomicOr(S.error, kErrStack); return kStDone; }
    uint32_t* top = stk + T.sp * stride;
    if (more > 2) { *top = (uint32_t)r3; top += stride; }
    if (more > 1) { *top = (uint32_t)r2; top += stride; }
    if (more > 0) *top = (uint32_t)r1;
    T.sp += more;
    return trav_next(T, t0 < inf ? r0 : kRefPop, stk, stride);
}

// Leaves the instance whose marker T.ref is and enters the next one, or enters instance T.ref.
GK_D int trav_trans(Trav& T, const SceneView& S, uint32_t* stk, int stride, int cap) {
    T.o = T.wo;
    T.d = T.wd;
    int st = kStTrans;
    if (T.ref == kRefMarker) {
        T.inblas = false;
        st = trav_next(T, kRefPop, stk, stride);
    }
    if (st == kStTrans) {
        T.cur = ~(uint32_t)T.ref >> 3;
        GK_CHECK_OR_END(T.cur < S.inst_count, S, T, kStDone);
        const DevInst* ip = S.inst + T.cur;
        float w[12];
        const int root = __ldg(&ip->blas_root);
        load_winv(ip, w);
        T.o = xpoint(w, T.wo);
        T.d = xvector(w, T.wd);
        if (T.sp >= cap) { atomicOr(S.error, kErrStack); return kStDone; }
        stk[T.sp * stride] = (uint32_t)kRefMarker;
        ++T.sp;
        T.inblas = true;
        T.ref = root;
        st = kStNode;
    }
    T.sl = quad_slabs(T.o, T.d);
    return st;
}

// Tests the triangles of leaf T.ref.
template <bool kRayTmin = false>
GK_D int trav_tris(Trav& T, const SceneView& S, const uint32_t* stk, int stride, Counters& cn) {
    const uint32_t leaf = ~(uint32_t)T.ref;
    GK_CHECK_OR_END((leaf >> 3) + (leaf & 7u) + 1u <= S.tri_count, S, T, kStDone);
    if (trav_leaf<kRayTmin>(T, S, leaf >> 3, (leaf & 7u) + 1u, cn)) return kStDone;
    return trav_next(T, kRefPop, stk, stride);
}

// t of byte `b` of `word` (a WideNode plane): fma(2^23 + q, C, B').
GK_D float wide_t(uint32_t word, int b, float C, float Bp) {
    return fmaf_(__uint_as_float(__byte_perm(word, 0x4B000000u, 0x7540u + (uint32_t)b)), C, Bp);
}

GK_D void wide_sort_cx(uint32_t& a, uint32_t& b) {
    const uint32_t lo = min(a, b);
    b = max(a, b);
    a = lo;
}

GK_D void trav_to_world(Trav& T) {
    T.o = T.wo; T.d = T.wd; T.inv = safe_inv(T.wd);
    T.inblas = false;
}

// Node phase of the traversal ("while-while", Aila and Laine, HPG 2009, over 8-wide nodes).
// The group stack holds one entry per wide node with more than one child left to visit:
// three words (node index or kRefMarker; pending slots; t lower bound). Pending word: bits
// 0-2 the count c of slots left, bits 3 + 3i the i-th slot to visit next, nearest first.
// A step pops (dropping groups whose nearest pending child lies beyond the current hit) and
// tests the popped node's eight children in the same call, so the lanes of a warp stay on
// the same instructions. A triangle leaf is postponed into T.leaf and the lane waits for the
// leaf phase; so does a lane about to leave the instance of its postponed leaf. Returns true
// while the lane can take another node step.
GK_D bool trav_node_step_wide(Trav& T, const SceneView& S, uint32_t* stk, int stride, Counters& cn) {
    if (++T.iter > kIterCap) { atomicOr(S.error, kErrIter); T.done = true; return false; }
    int ref = T.ref;
    if (ref == kRefMarker) {            // hand-back deferred until the postponed leaf was tested
        if (T.has_leaf) return false;
        trav_to_world(T);
        ref = kRefPop;
    }
    if (ref == kRefPop) {
        for (;;) {
            if (T.sp == 0) { T.done = true; T.ref = kRefPop; return false; }
            uint32_t* e = stk + 3 * (T.sp - 1) * stride;
            const uint32_t node = e[0];
            if (node == (uint32_t)kRefMarker) {
                --T.sp;
                if (T.has_leaf) { T.ref = kRefMarker; return false; }
                trav_to_world(T);
                continue;
            }
            const uint32_t w = e[stride];
            if (__uint_as_float(e[2 * stride]) > T.tcull) { --T.sp; continue; }
            GK_CHECK_OR_END(node < S.wide_count, S, T, false);
            const uint32_t c = w & 7u, slot = (w >> 3) & 7u;
            if (c <= 1u) --T.sp;
            else e[stride] = ((w >> 3) & ~7u) | (c - 1u);
            ref = __ldg(reinterpret_cast<const int*>(S.wide + node) + 16 + slot);
            break;
        }
    }
    if (ref >= 0) {
        GK_CHECK_OR_END((uint32_t)ref < S.wide_count, S, T, false);
        ++cn.nodes;
        const float4* np = reinterpret_cast<const float4*>(S.wide + ref);
        const float4 h = __ldg(np);
        const uint4 qx = __ldg(reinterpret_cast<const uint4*>(np + 1));
        const uint4 qy = __ldg(reinterpret_cast<const uint4*>(np + 2));
        const uint4 qz = __ldg(reinterpret_cast<const uint4*>(np + 3));
        const uint32_t meta = __float_as_uint(h.w);
        const float Cx = __uint_as_float((meta & 0xFFu) << 23) * T.inv.x;
        const float Cy = __uint_as_float(((meta >> 8) & 0xFFu) << 23) * T.inv.y;
        const float Cz = __uint_as_float(((meta >> 16) & 0xFFu) << 23) * T.inv.z;
        const float Bx = fmaf_(-8388608.0f, Cx, (h.x - T.o.x) * T.inv.x);
        const float By = fmaf_(-8388608.0f, Cy, (h.y - T.o.y) * T.inv.y);
        const float Bz = fmaf_(-8388608.0f, Cz, (h.z - T.o.z) * T.inv.z);
        // near / far plane words by the sign of the direction (the slab min / max)
        const bool nx = T.inv.x < 0.0f, ny = T.inv.y < 0.0f, nz = T.inv.z < 0.0f;
        const uint32_t nx0 = nx ? qx.z : qx.x, nx1 = nx ? qx.w : qx.y, fx0 = nx ? qx.x : qx.z, fx1 = nx ? qx.y : qx.w;
        const uint32_t ny0 = ny ? qy.z : qy.x, ny1 = ny ? qy.w : qy.y, fy0 = ny ? qy.x : qy.z, fy1 = ny ? qy.y : qy.w;
        const uint32_t nz0 = nz ? qz.z : qz.x, nz1 = nz ? qz.w : qz.y, fz0 = nz ? qz.x : qz.z, fz1 = nz ? qz.y : qz.w;
        uint32_t key[8];
        uint32_t nhit = 0;
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const int b = i & 3;
            const float tnx = wide_t(i < 4 ? nx0 : nx1, b, Cx, Bx), tfx = wide_t(i < 4 ? fx0 : fx1, b, Cx, Bx);
            const float tny = wide_t(i < 4 ? ny0 : ny1, b, Cy, By), tfy = wide_t(i < 4 ? fy0 : fy1, b, Cy, By);
            const float tnz = wide_t(i < 4 ? nz0 : nz1, b, Cz, Bz), tfz = wide_t(i < 4 ? fz0 : fz1, b, Cz, Bz);
            // slab interval widened by 1e-6 relative; T.tcull carries the same widening
            const float tn = fmaxf(fmaxf(tnx, tny), fmaxf(tnz, T.tmin));
            const float tf = fminf(fminf(tfx, tfy), tfz) * 1.000001f;
            const bool hit = ((meta >> (24 + i)) & 1u) && tn <= fminf(tf, T.tcull);
            key[i] = hit ? ((__float_as_uint(tn) & ~7u) | (uint32_t)i) : 0xFFFFFFFFu;
            nhit += hit ? 1u : 0u;
        }
        if (nhit == 0u) {
            T.ref = kRefPop;
            return true;
        }
        // Batcher's odd-even merge sort of the 8 keys (tnear bits, slot in the low bits)
        wide_sort_cx(key[0], key[1]); wide_sort_cx(key[2], key[3]); wide_sort_cx(key[4], key[5]);
        wide_sort_cx(key[6], key[7]); wide_sort_cx(key[0], key[2]); wide_sort_cx(key[1], key[3]);
        wide_sort_cx(key[4], key[6]); wide_sort_cx(key[5], key[7]); wide_sort_cx(key[1], key[2]);
        wide_sort_cx(key[5], key[6]); wide_sort_cx(key[0], key[4]); wide_sort_cx(key[1], key[5]);
        wide_sort_cx(key[2], key[6]); wide_sort_cx(key[3], key[7]); wide_sort_cx(key[2], key[4]);
        wide_sort_cx(key[3], key[5]); wide_sort_cx(key[1], key[2]); wide_sort_cx(key[3], key[4]);
        wide_sort_cx(key[5], key[6]);
        if (nhit > 1u) {
            if (T.sp >= kStackEntries) { atomicOr(S.error, kErrStack); T.done = true; return false; }
            uint32_t w = nhit - 1u;
#pragma unroll
            for (int j = 1; j < 8; ++j) w |= (key[j] & 7u) << (3 * j);
            uint32_t* e = stk + 3 * T.sp * stride;
            e[0] = (uint32_t)ref;
            e[stride] = w;
            e[2 * stride] = key[1] & ~7u;   // <= the nearest pending child's tnear
            ++T.sp;
        }
        const uint32_t s0 = key[0] & 7u;
        const int4 rr = __ldg(reinterpret_cast<const int4*>(np + 4 + (s0 >> 2)));
        ref = (s0 & 2u) ? ((s0 & 1u) ? rr.w : rr.z) : ((s0 & 1u) ? rr.y : rr.x);
        if (ref >= 0) {
            T.ref = ref;
            return true;
        }
        // nearest child is an instance or a triangle leaf: enter or postpone it here
    }
    const uint32_t payload = ~(uint32_t)ref;
    if (!T.inblas) {
        T.cur = payload >> 3;
        GK_CHECK_OR_END(T.cur < S.inst_count, S, T, false);
        const DevInst* ip = S.inst + T.cur;
        float w[12];
        load_winv(ip, w);
        T.o = xpoint(w, T.wo);
        T.d = xvector(w, T.wd);
        T.inv = safe_inv(T.d);
        if (T.sp >= kStackEntries) { atomicOr(S.error, kErrStack); T.done = true; return false; }
        uint32_t* e = stk + 3 * T.sp * stride;
        e[0] = (uint32_t)kRefMarker;
        e[stride] = 0u;
        e[2 * stride] = 0u;
        ++T.sp;
        T.inblas = true;
        T.ref = __ldg(&ip->blas_wide_root);
        return true;
    }
    if (T.has_leaf) {                   // one postponed leaf at a time
        T.ref = ref;
        return false;
    }
    T.leaf = payload;
    T.has_leaf = true;
    T.ref = kRefPop;
    return kSpeculative;
}

// Leaf phase: test the postponed leaf's triangles.
template <bool kRayTmin = false>
GK_D void trav_leaf_step(Trav& T, const SceneView& S, Counters& cn) {
    if (!T.has_leaf) return;
    GK_CHECK_OR_END((T.leaf >> 3) + (T.leaf & 7u) + 1u <= S.tri_count, S, T, );
    T.has_leaf = false;
    if (trav_leaf<kRayTmin>(T, S, T.leaf >> 3, (T.leaf & 7u) + 1u, cn)) T.done = true;
}

GK_D bool trav_finished(const Trav& T) { return T.done && !T.has_leaf; }

// Whole-ray traversal over the 8-wide nodes: hits with tmin <= t <= tmax.
template <int MODE>
GK_D TraceOut traverse_wide(const SceneView& S, f3 wo, f3 wd, float tmin, float tmax, uint32_t* stk, int stride,
                            Counters& cn) {
    Trav T;
    trav_init<true>(T, S, wo, wd, tmax, MODE, tmin);
    while (!trav_finished(T)) {
        while (!T.done && trav_node_step_wide(T, S, stk, stride, cn)) {
        }
        trav_leaf_step<true>(T, S, cn);
    }
    TraceOut R;
    R.hit = T.hit; R.ambiguous = false; R.inst = T.inst; R.prim = T.prim; R.tri = T.tri;
    return R;
}

// Float t and barycentrics of the winning triangle (the values shading uses).
struct HitShade { float t, b1, b2; };
GK_D HitShade hit_shade(const SceneView& S, f3 wo, f3 wd, uint32_t inst, uint32_t tri) {
    float w[12];
    load_winv(S.inst + inst, w);
    f3 o = xpoint(w, wo), d = xvector(w, wd);
    Shear sh = make_shear(d);
    f3 v0 = tri_v(S.tris, tri, 0), v1 = tri_v(S.tris, tri, 1), v2 = tri_v(S.tris, tri, 2);
    Fp32Hit f = fp32_test(o, sh, v0, v1, v2);
    HitShade h;
    if (f.kind == 1) { h.t = f.t; h.b1 = f.b1; h.b2 = f.b2; return h; }
    ExactHit x = exact_test(o, d, v0, v1, v2);
    h.t = (float)x.t; h.b1 = (float)x.b1; h.b2 = (float)x.b2;
    return h;
}

}  // namespace gk
