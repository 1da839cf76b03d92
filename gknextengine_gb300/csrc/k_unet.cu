// k_unet.cu — the learned denoiser's training and inference kernels besides the forward
// convolution (k_conv.cu): weight gradients on the tensor cores, and the element-wise part of each
// layer's backward pass.
//
// The weight gradient of a 3x3 convolution, dW[cout][tap][cin] = sum over pixels of
// dP[p][cout] * X[p + tap offset][cin], is a GEMM with K = pixels whose operands TMA loads
// straight from the NHWC tensors in the MN-major layout (k_conv_wgrad, below).
#include <algorithm>

#include "gk_umma.cuh"
#include "gkrt_internal.h"

namespace gk {

namespace {

// ---- weight gradient with TMA-fed MN-major operands ----
// dW[cout][tap][cin] = sum over pixels of dP[p][cout] X[p + tap][cin] with K = pixels: NHWC rows hold
// the channels of one pixel contiguously, which is the MN-major layout of both operands for K along
// pixels, so TMA loads them unchanged, 64-byte swizzled (atoms of 8 pixels x 64 bytes; an operand may
// start at any pixel of a box). All nine taps of 32 x 32 channels are one MMA of 128 x 96:
//   M  rows are the box of one 32-channel group of X, {32 channels, 34 pixels, 4 image rows}, at
//      pixel offsets 0, 1 and 2 (the taps dx): atoms one pixel apart. The fourth is not used;
//   N  columns are the dP rows r - 1, r, r + 1 of one 32-channel group against X's row r (the taps
//      dy = 1, 0, -1): consecutive rows of one box with a halo row on each side. At an image's first and
//      last row N leaves out the dP row outside it, whose zeros times an infinite X would be NaN in a tap
//      that this row has no part in; and X rows past the image take no MMA.
// So an X element is loaded once and a dP element 1.5 times. TMA's zero fill is the horizontal
// padding, and the channels past the tensors' ends. A CTA takes up to kWgCombos pairs of X and dP
// groups (their accumulators fill the 512 TMEM columns; they are zeroed first, 0.2 to 0.4 us a launch, and
// every MMA adds, whichever columns it covers) and a run of tiles; warp 0 issues the loads
// into a ring of stages, a lane to a box, warps 1 and 2 the MMAs of every other pair, and the
// warps 0-2 (dx) add the accumulators to dW: a warp's 32 lanes hold 32 consecutive input channels, and
// through shared memory each lane gets four of them for one 16-byte addition (a quarter of the
// additions at L2: 224 x 96 took 43.5 us with one value per addition, 39 with these; a dW that is not
// 16-byte aligned keeps the single ones). Every wait is bounded.
// What bounds it: the operand reads of shared memory (56 cycles an MMA) and the TMA unit (1.6 cycles a
// box row of 64 bytes).
// Before and after, on 8 x 256 x 256 pixels: 32 x 32 channels 119 us with one tap of one 64-channel atom
// per MMA, every operand read once per tap; 31 with four X boxes, each at its shift, as an M block; now
// 21. 96 x 32: 261, 90, 37. On 8 x 128 x 128: 64 x 64 75, 29, 22; on 8 x 64 x 64: 224 x 96 72, 39, 31.
// Of those now the additions to dW at L2 are 2 to 12 us. Tiles of 8 rows: 19, 40, 25, 25.

constexpr int kWtThreads = 128;
constexpr int kWgPix = 32;            // pixels of a tile row
constexpr int kWgXPix = kWgPix + 2;   // of X
constexpr int kWgRows = 4;            // X rows of a tile
constexpr int kWgXBox = kWgXPix * kWgRows * 64;        // 8.5 KB
constexpr int kWgDBox = kWgPix * (kWgRows + 2) * 64;   // 12 KB
constexpr int kWgCombos = 5;
constexpr int kWgSmem = 200 * 1024;   // stages
constexpr int kWgMaxStages = 6;
constexpr int kWgExtra = 1024 + 256 + 4 * 2048;   // alignment, barriers, the epilogue's exchange

// How the pairs of X and dP group are split over CTAs: mb x gb pairs per CTA.
struct WgPlan {
    int na, ng;        // X groups, dP groups in all
    int mb, gb;        // per CTA
    int stages;
    int xt, yt;        // tiles per image row, row tiles per image
    int items;         // tiles in all
    int groups, grid;  // of pairs, CTAs each
    int segs;          // partial sums per CTA: the accumulators are added to dW and restarted
    int vec;           // dW takes 16-byte additions (16-byte aligned; cin is a multiple of 16)
};

__device__ __forceinline__ void red_add4(float* p, float4 v) {
    asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(p), "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w)
                 : "memory");
}

__global__ void __launch_bounds__(kWtThreads) k_conv_wgrad(const __grid_constant__ CUtensorMap mdp,
                                                           const __grid_constant__ CUtensorMap mx, WgradArgs a, WgPlan p) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    const int stage_bytes = p.mb * kWgXBox + p.gb * kWgDBox;
    uint64_t* full = reinterpret_cast<uint64_t*>(smem + p.stages * stage_bytes);
    uint64_t* empty = full + kWgMaxStages;
    uint64_t* accb = empty + kWgMaxStages;
    uint32_t* tslot = reinterpret_cast<uint32_t*>(accb + 1);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tslot + 1);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    float* tb = reinterpret_cast<float*>(smem + p.stages * stage_bytes + 256) + warp * 512;   // 2 KB per warp
    const int msplit = (p.na + p.mb - 1) / p.mb;
    const int blk0 = ((int)blockIdx.y % msplit) * p.mb, g0 = ((int)blockIdx.y / msplit) * p.gb;
    const int nb = min(p.mb, p.na - blk0), ng = min(p.gb, p.ng - g0);
    const int i0 = (int)((long long)p.items * blockIdx.x / gridDim.x);
    const int i1 = (int)((long long)p.items * (blockIdx.x + 1) / gridDim.x);
    const int combos = p.mb * p.gb;
    const uint32_t ncols = combos == 1 ? 128u : combos == 2 ? 256u : 512u;

    if (tid == 0) {
        for (int st = 0; st < p.stages; ++st) {
            mbar_init(&full[st], 1);
            mbar_init(&empty[st], 2);   // both issuers
        }
        mbar_init(accb, 2);
        *abort_flag = 0;
        mbar_fence_init();
    }
    if (warp == 1) {
        tmem_alloc(tslot, ncols);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    grid_dep_launch();
    const uint32_t tmem = *tslot, mine = tmem + ((uint32_t)(warp * 32) << 16);   // this warp's lanes
    auto zero_pair = [&](int c) {
#pragma unroll
        for (int j = 0; j < 3; ++j) tmem_zero32(mine + (uint32_t)(96 * c + 32 * j));
    };
    if (warp < 3)   // (the fourth M block is not used)
        for (int c = 0; c < nb * ng; ++c) zero_pair(c);
    tmem_st_wait();
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    grid_dep_wait();

    // the producer's lane: its box's map, place in a stage, channels and offset from the tile's corner
    const bool is_x = lane < nb, loads = lane < nb + ng;
    const CUtensorMap* map = is_x ? &mx : &mdp;
    const int place = is_x ? lane * kWgXBox : p.mb * kWgXBox + (lane - nb) * kWgDBox;
    const int ch = 32 * (is_x ? blk0 + lane : g0 + lane - nb);
    int tx = 0, ty = 0, img = 0;   // the next tile's
    if (warp < 3) {
        const int per_img = p.xt * p.yt, rem = i0 % per_img;
        img = i0 / per_img;
        ty = rem / p.xt;
        tx = rem - ty * p.xt;
    }
    int s = 0;          // the next stage, and its uses so far
    uint32_t use = 0;

    for (int seg = 0; seg < p.segs; ++seg) {
        const int k0 = (int)((long long)(i1 - i0) * seg / p.segs), k1 = (int)((long long)(i1 - i0) * (seg + 1) / p.segs);
        if (warp == 0) {   // producer
            const uint32_t bytes = (uint32_t)(nb * kWgXBox + ng * kWgDBox);
            for (int k = k0; k < k1; ++k) {
                bool ok = !*abort_flag;
                if (use > 0) ok = mbar_wait_bounded(&empty[s], (use - 1u) & 1u, a.err) && ok;
                if (!__all_sync(0xFFFFFFFFu, ok)) {
                    *abort_flag = 1;
                    break;
                }
                if (lane == 0) mbar_expect_tx(&full[s], bytes);
                __syncwarp();
                if (loads)
                    tma_load_4d(smem + s * stage_bytes + place, map, ch, tx * kWgPix - (is_x ? 1 : 0),
                                ty * kWgRows - (is_x ? 0 : 1), img, &full[s]);
                if (++tx == p.xt) {
                    tx = 0;
                    if (++ty == p.yt) {
                        ty = 0;
                        ++img;
                    }
                }
                if (++s == p.stages) {
                    s = 0;
                    ++use;
                }
            }
        } else if (warp < 3) {   // MMA issuers
            constexpr uint32_t kHi = (512u >> 4) | (1u << 14) | (4u << 29);   // 8-pixel groups 512 bytes apart, SWIZZLE_64B
            const bool leader = elect_one();
            const uint32_t idesc = umma_idesc_bf16(128u, 96u) | (1u << 15) | (1u << 16);   // MN-major A, B
            constexpr uint32_t kDRow = kWgPix * 64 / 16;   // a row of a dP box
            const uint32_t base = smem_u32(smem) >> 4;
            bool ok = true;
            for (int k = k0; k < k1; ++k) {
                const int rows = a.H - ty * kWgRows;   // of the image, from the tile's first on
                const bool inner = ty > 0 && rows > kWgRows;
                ok = __all_sync(0xFFFFFFFFu, mbar_wait_bounded(&full[s], use & 1u, a.err));
                if (!ok) {
                    *abort_flag = 1;
                    break;
                }
                tc_fence_after();
                if (leader) {
                    // atoms along M: one pixel apart; along N: one dP row apart
                    const uint32_t st = base + (uint32_t)(s * (stage_bytes >> 4));
                    const uint32_t sx = st | ((64u >> 4) << 16), sd = (st + (uint32_t)(p.mb * (kWgXBox >> 4))) |
                                                                      (kDRow << 16);
                    if (inner) {
                        for (int m = 0, c = 0; m < nb; ++m)
                            for (int g = 0; g < ng; ++g, ++c) {
                                if ((c & 1) != warp - 1) continue;
                                const uint32_t d = tmem + (uint32_t)(c * 96);
                                const uint32_t al = sx + (uint32_t)(m * (kWgXBox >> 4)), bl = sd + (uint32_t)(g * (kWgDBox >> 4));
                                auto mma = [&](int r, uint32_t dd, uint32_t bb, uint32_t id) {   // 16 pixels (two 8-pixel groups)
                                    umma_bf16_lo(dd, al + (uint32_t)((r >> 1) * (kWgXPix * 4) + (r & 1) * 64), kHi,
                                                 bb + (uint32_t)(r * 64), kHi, id, 1u);
                                };
#pragma unroll
                                for (int r = 0; r < 2 * kWgRows; ++r) mma(r, d, bl, idesc);
                            }
                    } else {
                        // the image's first row has no dP row above, its last none below: 32 columns less (N / 8
                        // starts at bit 17). A loop of its own: with these operands in registers for every tile
                        // 96 x 32 channels on 2 x 509 x 517 pixels took 42.0 us; 41.0 so, as before the outer rows
                        // were told apart
                        const uint32_t up = ty == 0 ? 1u : 0u, down = rows == kWgRows ? 1u : 0u;
                        const uint32_t id0 = idesc - (up << 19), id3 = idesc - (down << 19), up_d = up * 32u, up_b = up * kDRow;
                        for (int m = 0, c = 0; m < nb; ++m)
                            for (int g = 0; g < ng; ++g, ++c) {
                                if ((c & 1) != warp - 1) continue;
                                const uint32_t d = tmem + (uint32_t)(c * 96);
                                const uint32_t al = sx + (uint32_t)(m * (kWgXBox >> 4)), bl = sd + (uint32_t)(g * (kWgDBox >> 4));
                                auto mma = [&](int r, uint32_t dd, uint32_t bb, uint32_t id) {
                                    umma_bf16_lo(dd, al + (uint32_t)((r >> 1) * (kWgXPix * 4) + (r & 1) * 64), kHi,
                                                 bb + (uint32_t)(r * 64), kHi, id, 1u);
                                };
                                if (rows >= kWgRows) {
                                    mma(0, d + up_d, bl + up_b, id0);
                                    mma(1, d + up_d, bl + up_b, id0);
                                    mma(2, d, bl, idesc);
                                    mma(3, d, bl, idesc);
                                    mma(4, d, bl, idesc);
                                    mma(5, d, bl, idesc);
                                    mma(6, d, bl, id3);
                                    mma(7, d, bl, id3);
                                } else {
                                    for (int r = 0; r < 2 * rows; ++r) {
                                        const uint32_t u = r < 2 ? up : 0u;
                                        mma(r, d + 32u * u, bl + kDRow * u,
                                            idesc - ((u + ((r >> 1) == rows - 1 ? 1u : 0u)) << 19));
                                    }
                                }
                            }
                    }
                    umma_commit(&empty[s]);
                }
                __syncwarp();
                if (++tx == p.xt) {
                    tx = 0;
                    if (++ty == p.yt) ty = 0;
                }
                if (++s == p.stages) {
                    s = 0;
                    ++use;
                }
            }
            if (leader) umma_commit(accb);
            __syncwarp();
        }
        __syncwarp();
        const bool summed = mbar_wait_bounded(accb, (uint32_t)seg & 1u, a.err);
        if (!summed) *abort_flag = 1;
        const bool ready = __all_sync(0xFFFFFFFFu, summed && k1 > k0 && !*abort_flag) != 0;
        tc_fence_after();
        // lane `lane` of warp dx: input channel 32 (blk0 + m) + lane
        const int dx = warp;
        for (int part = 0; part < nb * ng * 6; ++part) {
            const int c = part / 6, n0 = (part - 6 * c) * 16, m = c / ng, g = c - m * ng;
            const int ci = 32 * (blk0 + m) + lane;
            uint32_t v[16];
            tmem_ld16(tmem + ((uint32_t)(warp * 32) << 16) + (uint32_t)(c * 96 + n0), v);
            tmem_ld_wait();
            if (seg + 1 < p.segs && n0 == 80) zero_pair(c);   // all six parts have been read
            if (!ready || dx > 2) continue;   // the same for the whole warp
            const int dy = 2 - n0 / 32;   // tap row: dP's row r - 1 is tap dy = +1
            const int co = 32 * (g0 + g) + (n0 & 31);
            float* d = a.dw + ((size_t)co * 9 + 3 * dy + dx) * a.cin + (ci - lane);
            if (p.vec) {   // 16 x 32 values as four consecutive input channels per lane and addition
#pragma unroll
                for (int j = 0; j < 16; ++j) tb[j * 32 + lane] = __uint_as_float(v[j]);
                __syncwarp();
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const int r = 4 * j + (lane >> 3), c4 = 4 * (lane & 7);
                    const float4 f = *reinterpret_cast<const float4*>(tb + r * 32 + c4);
                    if (co + r < a.cout && ci - lane + c4 < a.cin) red_add4(d + (size_t)r * 9 * a.cin + c4, f);
                }
                __syncwarp();
            } else if (ci < a.cin) {
#pragma unroll
                for (int j = 0; j < 16; ++j) {
                    const float f = __uint_as_float(v[j]);
                    if (f != 0.0f && co + j < a.cout) atomicAdd(d + lane + (size_t)j * 9 * a.cin, f);
                }
            }
        }
        tmem_st_wait();
        tc_fence_before();
        if (__syncthreads_or(*abort_flag)) break;   // the next sums start in the accumulators read here
        tc_fence_after();
    }
    if (warp == 0)   // no load may be in flight when the CTA ends, whoever gave up
        for (int i = 0; i < p.stages; ++i) {
            const uint32_t uses = use + (i < s ? 1u : 0u);
            if (uses > 0) mbar_wait_bounded(&full[i], (uses - 1u) & 1u, a.err);
        }
    __syncthreads();
    if (warp == 1) tmem_dealloc(tmem, ncols);
}

// ---- element-wise kernels (NHWC bf16 with channel stride/offset) ----
// One thread per pixel and group of 8 channels (16-byte loads and stores); channel counts,
// strides and offsets are multiples of 8. Pixel counts fit 32-bit indices.

__device__ __forceinline__ void ld8(const __nv_bfloat16* p, float* v) {
    const uint4 u = *reinterpret_cast<const uint4*>(p);
    const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&u);
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const float2 f = __bfloat1622float2(h[k]);
        v[2 * k] = f.x;
        v[2 * k + 1] = f.y;
    }
}
__device__ __forceinline__ void st8(__nv_bfloat16* p, const float* v) {
    uint4 u;
    __nv_bfloat162* h = reinterpret_cast<__nv_bfloat162*>(&u);
#pragma unroll
    for (int k = 0; k < 4; ++k) h[k] = __floats2bfloat162_rn(v[2 * k], v[2 * k + 1]);
    *reinterpret_cast<uint4*>(p) = u;
}

// One layer's gradient of its pre-activation, dP = dY * (Y > 0), in place of dY, and its bias
// gradient db[c] += sum over pixels of dP[p][c], in one pass over dY; and on the way there what dY
// is still to receive:
//   kPool      dY += d_pool / 4 of the half-resolution pixel (the 2 x 2 average pooling's gradient);
//   kUpsample  dY = sum of the 2 x 2 double-resolution gradients it was copied to;
// each rounded to bf16 before the ReLU's mask, as a pass of its own would store it. y null: no ReLU.
// One block per run of pixels. Thread t owns the 8 channels 8 (t % G) .. +7 (G = C / 8, 16-byte
// loads and stores) of every (256 / G)-th pixel of the run and sums them in registers; the threads
// of each channel group are then reduced in shared memory and each channel gets one atomic per
// block. Three separate passes and a run of 1024 pixels per block (8 blocks for the eighth-resolution
// layers) took 0.45 ms of an 8 x 256 x 256 training step; now 0.13.
enum GradMode { kGradPlain = 0, kGradPool = 1, kGradUpsample = 2 };
template <int kMode>
__global__ void __launch_bounds__(256) k_layer_grad(LayerGradArgs a, int run) {
    __shared__ float part[256 * 8];
    grid_dep_launch();
    grid_dep_wait();
    const int G = a.C / 8, per = 256 / G;
    const int g = threadIdx.x % G, k = threadIdx.x / G;
    float acc[8] = {0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f};
    if (k < per) {
        const int p0 = blockIdx.x * run, p1 = min(p0 + run, a.B * a.H * a.W);
        for (int p = p0 + k; p < p1; p += per) {
            float v[8];
            __nv_bfloat16* d = a.dy + (size_t)p * a.dy_c + a.dy_off + 8 * g;
            if (kMode == kGradUpsample) {
                const int x = p % a.W, y = (p / a.W) % a.H, b = p / (a.W * a.H);
                float t[8];
#pragma unroll
                for (int j = 0; j < 8; ++j) v[j] = 0.0f;
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    const size_t s = (size_t)(b * 2 * a.H + 2 * y + (q >> 1)) * (2 * a.W) + 2 * x + (q & 1);
                    ld8(a.src + s * a.src_c + a.src_off + 8 * g, t);
#pragma unroll
                    for (int j = 0; j < 8; ++j) v[j] += t[j];
                }
            } else {
                ld8(d, v);
                if (kMode == kGradPool) {
                    const int x = p % a.W, y = (p / a.W) % a.H, b = p / (a.W * a.H);
                    const size_t s = (size_t)(b * (a.H / 2) + y / 2) * (a.W / 2) + x / 2;
                    float t[8];
                    ld8(a.src + s * a.src_c + a.src_off + 8 * g, t);
#pragma unroll
                    for (int j = 0; j < 8; ++j) v[j] = 0.25f * t[j] + v[j];
                }
            }
            if (kMode != kGradPlain) {
#pragma unroll
                for (int j = 0; j < 8; ++j) v[j] = __bfloat162float(__float2bfloat16_rn(v[j]));
            }
            if (a.y) {
                float y8[8];
                ld8(a.y + (size_t)p * a.y_c + a.y_off + 8 * g, y8);
#pragma unroll
                for (int j = 0; j < 8; ++j)
                    if (!(y8[j] > 0.0f)) v[j] = 0.0f;
            }
            if (a.y || kMode != kGradPlain) st8(d, v);
#pragma unroll
            for (int j = 0; j < 8; ++j) acc[j] += v[j];
        }
    }
#pragma unroll
    for (int j = 0; j < 8; ++j) part[threadIdx.x * 8 + j] = acc[j];
    __syncthreads();
    if (threadIdx.x < a.C) {
        const int c = threadIdx.x, cg = c / 8, cj = c % 8;
        float sum = 0.0f;
        for (int i = 0; i < per; ++i) sum += part[(i * G + cg) * 8 + cj];
        if (sum != 0.0f) atomicAdd(&a.db[c], sum);
    }
}

}  // namespace

}  // namespace gk

using namespace gk;

cudaError_t gkrt_encode_tmap_bf16(CUtensorMap* map, const void* base, uint32_t rank, const uint64_t* dims,
                                  const uint64_t* strides_bytes, const uint32_t* box);

// The split with the fewest cycles a tile, over all groups of pairs: MMAs, or box rows if those are more. At
// least two stages (a box of X per group, and one of dP, 1.5 times as tall) fit in shared memory.
static WgPlan wgrad_plan(const WgradArgs& a, int sms) {
    WgPlan p{};
    p.na = (a.cin + 31) / 32;
    p.ng = (a.cout + 31) / 32;
    double best = 1e30;
    for (int mb = 1; mb <= std::min(p.na, kWgCombos); ++mb)
        for (int gb = 1; gb <= std::min(p.ng, kWgCombos / mb); ++gb) {
            const int bytes = mb * kWgXBox + gb * kWgDBox;
            if (2 * bytes > kWgSmem) continue;
            const int groups = ((p.na + mb - 1) / mb) * ((p.ng + gb - 1) / gb);
            const double cost = groups * (150.0 + std::max(mb * gb * kWgRows * 2 * 56.0, bytes / 64 * 1.6));
            if (cost < best) {
                best = cost;
                p.mb = mb;
                p.gb = gb;
                p.stages = std::min(kWgMaxStages, kWgSmem / bytes);
            }
        }
    p.xt = (a.W + kWgPix - 1) / kWgPix;
    p.yt = (a.H + kWgRows - 1) / kWgRows;
    p.items = a.B * p.xt * p.yt;
    p.vec = ((uintptr_t)a.dw & 15u) == 0u;
    p.groups = ((p.na + p.mb - 1) / p.mb) * ((p.ng + p.gb - 1) / p.gb);
    // one CTA per SM (its stages fill the shared memory), at least two tiles each. From 136 tiles on an FP32
    // sum covers at most a 34th of the pixels: with 21 CTAs, 224 x 96 on 8 x 64 x 64 was off by 1.6e-6 of dW's
    // norm in one sum each (25 us) and is by 7.4e-7 in two (31 us). (Fewer tiles are at most 17,280 pixels
    // in all: a sum may cover more than a 34th of them, of fewer terms.)
    p.grid = std::max(1, std::min((p.items + 1) / 2, sms / p.groups));
    p.segs = p.items < 34 * 4 ? 1 : (34 + p.grid - 1) / p.grid;
    return p;
}
// For the tests: the partial sums of each CTA, on a device of `sms`.
extern "C" int gkrt_internal_wgrad_sums(int B, int H, int W, int cin, int cout, int sms) {
    WgradArgs a{};
    a.B = B; a.H = H; a.W = W; a.cin = cin; a.cout = cout;
    return wgrad_plan(a, sms).segs;
}

cudaError_t gkrt_launch_conv_wgrad(const WgradArgs& a, cudaStream_t st) {
    const int xv = a.x_valid > 0 ? a.x_valid : a.cin;   // X's channels present; the rest are zeros
    if (a.cin % 16 || a.cin < 16 || a.cin > 256 || a.cout % 8 || a.cout < 8 || a.cout > 128 || a.dp_c % 8 ||
        a.dp_off % 8 || a.x_c % 8 || a.x_off % 8 || a.dp_off + a.cout > a.dp_c || a.x_valid < 0 ||
        a.x_valid > a.cin || a.x_valid % 8 || a.x_off + xv > a.x_c || ((uintptr_t)a.dp & 15u) ||
        ((uintptr_t)a.x & 15u) || a.B < 1 || a.H < 1 || a.W < 1)
        return cudaErrorInvalidValue;
    if ((long long)a.B * ((a.W + kWgPix - 1) / kWgPix) * ((a.H + kWgRows - 1) / kWgRows) > 0x7FFFFFFFLL)
        return cudaErrorInvalidValue;
    static int sms_dev[kMaxDevices] = {};
    const int dev = current_device_slot();
    if (dev < 0) return cudaErrorInvalidDevice;
    if (!sms_dev[dev]) {
        cudaError_t e = cudaFuncSetAttribute(k_conv_wgrad, cudaFuncAttributeMaxDynamicSharedMemorySize, kWgSmem + kWgExtra);
        if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms_dev[dev], cudaDevAttrMultiProcessorCount, dev);
        if (e != cudaSuccess) return e;
    }
    const uint64_t W = (uint64_t)a.W, H = (uint64_t)a.H, B = (uint64_t)a.B;
    const WgPlan p = wgrad_plan(a, sms_dev[dev]);
    const uint32_t dbox[4] = {32u, (uint32_t)kWgPix, (uint32_t)(kWgRows + 2), 1u};
    const uint32_t xbox[4] = {32u, (uint32_t)kWgXPix, (uint32_t)kWgRows, 1u};
    CUtensorMap mdp, mx;
    const uint64_t dd[4] = {(uint64_t)a.cout, W, H, B};
    const uint64_t ds[3] = {(uint64_t)a.dp_c * 2, W * a.dp_c * 2, H * W * a.dp_c * 2};
    cudaError_t e = gkrt_encode_tmap_bf16(&mdp, a.dp + a.dp_off, 4, dd, ds, dbox);
    if (e != cudaSuccess) return e;
    const uint64_t xd[4] = {(uint64_t)xv, W, H, B};   // channels past xv: TMA's zero fill
    const uint64_t xs[3] = {(uint64_t)a.x_c * 2, W * a.x_c * 2, H * W * a.x_c * 2};
    if ((e = gkrt_encode_tmap_bf16(&mx, a.x + a.x_off, 4, xd, xs, xbox)) != cudaSuccess) return e;
    const int stage_bytes = p.mb * kWgXBox + p.gb * kWgDBox;
    return launch_after(k_conv_wgrad, dim3((unsigned)p.grid, (unsigned)p.groups), kWtThreads,
                        (size_t)p.stages * stage_bytes + kWgExtra, st, mdp, mx, a, p);
}

cudaError_t gkrt_launch_layer_grad(const LayerGradArgs& a, int mode, cudaStream_t st) {
    const long long npix = (long long)a.B * a.H * a.W;
    if (a.C > 128 || a.C % 8 || a.C < 8 || a.dy_c % 8 || a.dy_off % 8 || ((uintptr_t)a.dy & 15u) ||
        npix > 0x7FFFFFFFLL / 4)
        return cudaErrorInvalidValue;
    // about four blocks per SM, each thread at least four pixels
    const int per = 256 / (a.C / 8);
    const int run = (int)std::max<long long>(4 * per, (npix + 607) / 608);
    const unsigned blocks = (unsigned)((npix + run - 1) / run);
    const auto kernel = mode == kGradPool       ? k_layer_grad<kGradPool>
                        : mode == kGradUpsample ? k_layer_grad<kGradUpsample>
                                                : k_layer_grad<kGradPlain>;
    kernel<<<blocks, 256, 0, st>>>(a, run);
    return cudaGetLastError();
}
