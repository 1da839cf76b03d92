// k_conv.cu — 3x3 "same" convolution as an implicit GEMM on the tcgen05 tensor cores.
//
// Building block of the learned denoiser (no counterpart in the reference, whose learned
// denoiser is the closed OIDN library). Activations are NHWC bf16 with channel counts that
// are multiples of 32; weights are [Cout][3][3][Cin] bf16; accumulation is FP32 in tensor
// memory.
//
// Four kernels, all persistent and warp-specialised, that take the FP32 sums of an output in the same
// order: k_conv_rows (row tiles, weights in shared memory) for the layers whose weights fit and whose
// images are large enough, k_conv_tiles (16 x 16 tiles, weights streamed) for the others of up to 128
// channels, and for the rest k_conv3x3_halo (outputs of up to 32 channels) and k_conv3x3,
// whose CTAs loop over tiles of 16 x 8 pixels (x by y, M = 128) times all Cout (N <= 256) of one image:
//   K loop   9 taps x Cin / 32 chunks. For tap (dy, dx) and chunk c the A operand is the
//            4D TMA box {32 channels, 16 x, 8 y, 1 image} of the input shifted by the tap;
//            coordinates outside the image read zeros, which is the zero padding. The B
//            operand is the 2D box {32, Cout} of the weights at column tap * Cin + 32 c.
//            Both land 64-byte swizzled, the K-major layout of gk_umma.cuh.
//   rows     for outputs of up to 128 channels (the full-resolution layers especially, whose few
//            MMAs per loaded byte leave them bound by L2 reads of the nine shifted boxes) one stage
//            holds the box {32, 16 x, 10 y, 1} at horizontal shift dx and the three weight
//            boxes of taps (0..2, dx): the three vertical taps are the windows starting 0, 1
//            and 2 image rows (1024 bytes, a whole number of 64-byte swizzle atoms) into the
//            box, so each input chunk is read 3 times instead of 9.
//   stages   warp 0 issues the TMA loads into a ring of shared-memory stages (full barriers
//            with transaction counts) across tile boundaries; warp 1 issues two K = 16 MMAs per
//            stage, frees the stage with tcgen05.commit (empty barriers) and commits each
//            tile's accumulator; two accumulators in TMEM alternate between tiles, so the
//            epilogue of one tile runs under the MMAs of the next.
//   epilogue warps 2-5 (one per TMEM lane quarter) read their 32 lanes (pixels) 16 columns at
//            a time, add the bias (and an optional half-resolution parity addend), apply ReLU,
//            store bf16 (or fp32) NHWC at a channel offset of a wider tensor (skip connections
//            are concatenated without copies; bf16 through the warp's shared-memory exchange,
//            whole 32-byte sectors per store), optionally with the 2 x 2 average and the
//            nearest upsampling, and release the accumulator.
// The grid holds as many CTAs per SM as shared memory and the 512 TMEM columns allow.
// Every barrier wait is bounded; a wait that runs out records the wait error bit in the
// device error word and the CTA skips its stores.
#include <algorithm>
#include <numeric>

#include <cuda_bf16.h>

#include "gk_umma.cuh"
#include "gkrt_internal.h"

namespace gk {

namespace {

constexpr int kConvThreads = 192;   // warp 0 TMA, warp 1 MMA, warps 2-5 epilogue
constexpr int kEpiThreads = 128;
constexpr int kTileX = 16, kTileY = 8;

__device__ __forceinline__ uint32_t pack_bf16x2(float a, float b) {
    const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<const uint32_t*>(&h);
}

// Shared memory of the bf16 epilogue: 1 KB per epilogue warp (16-byte aligned).
constexpr int kEpiBuf = 4 * 1024 + 16;

__device__ __forceinline__ size_t shfl_size(size_t v, int src) {
    const uint32_t lo = __shfl_sync(0xFFFFFFFFu, (uint32_t)v, src);
    const uint32_t hi = __shfl_sync(0xFFFFFFFFu, (uint32_t)((uint64_t)v >> 32), src);
    return (size_t)(((uint64_t)hi << 32) | lo);
}

// The bf16 epilogue of 16 channels (c0 .. c0 + 15) of pixel (x, y) of image img: the plain
// store, and the optional pooled and upsampled outputs. Called by every lane of the warp
// (the pool's 2 x 2 block is four lanes of one warp: x-neighbour lane ^ 1, y-neighbour lane ^
// yl); the pooled average is (((0 + v(x, y)) + v(x + 1, y)) + v(x, y + 1)) + v(x + 1, y + 1) of
// the stored (bf16-rounded) values, times 1/4, rounded to bf16. The warp's 32 pixels pass their
// 32 bytes through ebuf (this warp's 1 KB of shared memory; 16-byte chunks swizzled by lane bit
// 2, so that neither side has bank conflicts), and each 32-byte sector of the output is then
// written whole by two lanes of one store instruction: lane-per-pixel stores wrote every sector
// in two 16-byte halves from separate instructions, twice the L2 write requests.
// Where a lane's stores of one tile go, the same for every channel group (computed once per
// tile): the two pixels whose 16-byte halves it stores (element offsets into out and, for the
// nearest upsampling, of the top-left of the 2 x 2 block in up), and the pooled pixel whose
// four channels it stores.
struct EpiDst {
    size_t o[2], u[2], p;
    bool in[2], pin;
};
__device__ __forceinline__ EpiDst epi_dst(const ConvArgs& a, int img, int x, int y, bool inside, int yl) {
    const int lane = threadIdx.x & 31, h = lane & 1;
    const size_t pix = ((size_t)img * a.H + y) * a.W + x;
    const size_t uq = ((size_t)img * 2 * a.H + 2 * (size_t)y) * (2 * (size_t)a.W) + 2 * (size_t)x;
    EpiDst d;
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        const int src = (lane >> 1) + 16 * i;
        d.o[i] = shfl_size(pix, src) * a.out_c + a.out_off + 8 * h;
        d.in[i] = __shfl_sync(0xFFFFFFFFu, inside ? 1 : 0, src) != 0;
        d.u[i] = a.up_out ? shfl_size(uq, src) * a.up_c + a.up_off + 8 * h : 0;
    }
    d.p = 0;
    d.pin = false;
    if (a.pool_out) {
        const int h2 = a.H / 2, w2 = a.W / 2;
        const int b = yl == 16 ? 4 : 3;
        const int k = lane >> 2;
        const int tl = ((k >> (b - 1)) << (b + 1)) | ((k & ((1 << (b - 1)) - 1)) << 1);   // top-left lane
        const size_t pp = ((size_t)img * h2 + y / 2) * w2 + x / 2;
        const bool pvalid = !(x & 1) && !(y & 1) && x / 2 < w2 && y / 2 < h2;
        d.p = shfl_size(pp, tl) * a.pool_c + a.pool_off + 4 * (lane & 3);
        d.pin = __shfl_sync(0xFFFFFFFFu, pvalid ? 1 : 0, tl) != 0;
    }
    return d;
}

// The bf16 epilogue of 16 channels (c0 .. c0 + 15) of the warp's 32 pixels: the plain store,
// and the optional pooled and upsampled outputs. Called by every lane of the warp (the pool's
// 2 x 2 block is four lanes of one warp: x-neighbour lane ^ 1, y-neighbour lane ^ yl); the
// pooled average is (((0 + v(x, y)) + v(x + 1, y)) + v(x, y + 1)) + v(x + 1, y + 1) of the
// stored (bf16-rounded) values, times 1/4, rounded to bf16. The warp's 32 pixels pass their
// 32 bytes through ebuf (this warp's 1 KB of shared memory; 16-byte chunks swizzled by lane bit
// 2, so that neither side has bank conflicts), and each 32-byte sector of the output is then
// written whole by two lanes of one store instruction: lane-per-pixel stores wrote every sector
// in two 16-byte halves from separate instructions, twice the L2 write requests.
__device__ __forceinline__ void epilogue_bf16(const ConvArgs& a, const float (&v)[16], const EpiDst& d, int c0,
                                              int yl, uint4* ebuf) {
    const int lane = threadIdx.x & 31;
    const int sw = (lane >> 2) & 1;
    ebuf[2 * lane + sw] = make_uint4(pack_bf16x2(v[0], v[1]), pack_bf16x2(v[2], v[3]), pack_bf16x2(v[4], v[5]),
                                     pack_bf16x2(v[6], v[7]));
    ebuf[2 * lane + (sw ^ 1)] = make_uint4(pack_bf16x2(v[8], v[9]), pack_bf16x2(v[10], v[11]),
                                           pack_bf16x2(v[12], v[13]), pack_bf16x2(v[14], v[15]));
    __syncwarp();
    const size_t W2 = 2 * (size_t)a.W;
    const int h = lane & 1;
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        const int src = (lane >> 1) + 16 * i;
        const uint4 val = ebuf[2 * src + (h ^ ((src >> 2) & 1))];
        if (d.in[i]) *reinterpret_cast<uint4*>(reinterpret_cast<__nv_bfloat16*>(a.out) + d.o[i] + c0) = val;
        if (a.up_out && d.in[i]) {
            __nv_bfloat16* up = reinterpret_cast<__nv_bfloat16*>(a.up_out) + d.u[i] + c0;
            for (int k = 0; k < 4; ++k)
                *reinterpret_cast<uint4*>(up + ((k >> 1) * W2 + (k & 1)) * a.up_c) = val;
        }
    }
    __syncwarp();   // the next group rewrites ebuf
    if (a.pool_out) {
        // The warp's 8 pooled pixels x 16 channels: lane l averages channels 4 (l & 3) .. + 3 of
        // pooled pixel l >> 2 from the block's four stored values in ebuf (the block's top-left
        // lane, even x and even y, has lane bits 0 and log2(yl) clear; then its x-, y- and
        // diagonal neighbours, in that order) and stores them: 4 lanes per 32-byte sector.
        const int b = yl == 16 ? 4 : 3;
        const int k = lane >> 2, qd = lane & 3;
        const int tl = ((k >> (b - 1)) << (b + 1)) | ((k & ((1 << (b - 1)) - 1)) << 1);   // top-left lane
        float s4[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
        for (int t = 0; t < 4; ++t) {
            const int nl = tl ^ (t & 1) ^ (t & 2 ? yl : 0);
            const uint2 w = *reinterpret_cast<const uint2*>(reinterpret_cast<const uint8_t*>(ebuf) +
                                                            (2 * nl + ((qd >> 1) ^ ((nl >> 2) & 1))) * 16 +
                                                            (qd & 1) * 8);
            s4[0] = s4[0] + __uint_as_float(w.x << 16);
            s4[1] = s4[1] + __uint_as_float(w.x & 0xFFFF0000u);
            s4[2] = s4[2] + __uint_as_float(w.y << 16);
            s4[3] = s4[3] + __uint_as_float(w.y & 0xFFFF0000u);
        }
        if (d.pin)
            *reinterpret_cast<uint2*>(reinterpret_cast<__nv_bfloat16*>(a.pool_out) + d.p + c0) =
                make_uint2(pack_bf16x2(s4[0] * 0.25f, s4[1] * 0.25f), pack_bf16x2(s4[2] * 0.25f, s4[3] * 0.25f));
        __syncwarp();   // the next group rewrites ebuf
    }
}

// v[j] += bias[c0 + j] (bias null: nothing) as four 16-byte loads (the bias is 16-byte aligned).
__device__ __forceinline__ void add_bias16(const float* bias, int c0, float (&v)[16]) {
    if (!bias) return;
    const float4* b4 = reinterpret_cast<const float4*>(bias + c0);
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const float4 b = __ldg(b4 + k);
        v[4 * k] += b.x; v[4 * k + 1] += b.y; v[4 * k + 2] += b.z; v[4 * k + 3] += b.w;
    }
}

// The addend's 16 channels for output channels c0 .. c0 + 15 of pixel (x, y) (add_par): q is
// the element index of the half-resolution pixel's parity group.
__device__ __forceinline__ size_t pix_add(const ConvArgs& a, int img, int x, int y) {
    const size_t hp = ((size_t)img * (a.H >> 1) + (y >> 1)) * (a.W >> 1) + (x >> 1);
    return hp * a.add_c + (size_t)(((y & 1) << 1) | (x & 1)) * a.cout;
}
__device__ __forceinline__ void add_parity(const ConvArgs& a, float (&v)[16], size_t q, int c0) {
    const uint4* s = reinterpret_cast<const uint4*>(reinterpret_cast<const __nv_bfloat16*>(a.add_par) + q + c0);
    const uint4 lo = __ldg(s), hi = __ldg(s + 1);
    const uint32_t w[8] = {lo.x, lo.y, lo.z, lo.w, hi.x, hi.y, hi.z, hi.w};
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        v[2 * j] += __uint_as_float(w[j] << 16);
        v[2 * j + 1] += __uint_as_float(w[j] & 0xFFFF0000u);
    }
}

// fp32 output of channels c0 .. c0 + n - 1 (n <= 16) at o: 16-byte stores where o allows.
// Unrolled with constant indices, so that v stays in registers.
__device__ __forceinline__ void store_f32(float* o, const float (&v)[16], int n) {
    const bool al = !(reinterpret_cast<uintptr_t>(o) & 15u);
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        if (al && 4 * q + 4 <= n) {
            *reinterpret_cast<float4*>(o + 4 * q) = make_float4(v[4 * q], v[4 * q + 1], v[4 * q + 2], v[4 * q + 3]);
        } else {
#pragma unroll
            for (int j = 4 * q; j < 4 * q + 4; ++j)
                if (j < n) o[j] = v[j];
        }
    }
}

__device__ __forceinline__ void tile_origin(int t, int tiles_x, int tiles_y, int& x0, int& y0, int& img) {
    const int per_img = tiles_x * tiles_y;
    img = t / per_img;
    const int r = t - img * per_img;
    y0 = (r / tiles_x) * kTileY;
    x0 = (r % tiles_x) * kTileX;
}

// kRows: row-box stages (three vertical taps per stage) or one tap per stage. The MMA issuer
// adds each operand's offset to the descriptors' start fields as a constant.
template <bool kRows>
__global__ void __launch_bounds__(kConvThreads) k_conv3x3(const __grid_constant__ CUtensorMap mx,
                                                          const __grid_constant__ CUtensorMap mw, ConvArgs a,
                                                          int tiles_x, int tiles_y, int ntiles, int stages) {
    constexpr bool rows = kRows;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    const int a_bytes = kTileX * (rows ? kTileY + 2 : kTileY) * 64;
    const int b_bytes = a.cout * 64;
    constexpr int nb = rows ? 3 : 1;   // weight boxes per stage
    const int stage_bytes = (a_bytes + nb * b_bytes + 1023) & ~1023;
    uint64_t* full = reinterpret_cast<uint64_t*>(smem + stages * stage_bytes);
    uint64_t* empty = full + stages;
    uint64_t* accf = empty + stages;   // accumulator ready (MMA commit)
    uint64_t* acce = accf + 2;         // accumulator drained (128 epilogue arrivals)
    uint64_t* fin = acce + 2;          // every MMA of this CTA completed
    uint32_t* tslot = reinterpret_cast<uint32_t*>(fin + 1);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tslot + 1);
    uint4* ebuf = reinterpret_cast<uint4*>((reinterpret_cast<uintptr_t>(tslot + 2) + 15) & ~(uintptr_t)15);

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int kc = a.cin / 32, nk = (rows ? 3 : 9) * kc;
    const uint32_t ncols1 = a.cout <= 32 ? 32u : a.cout <= 64 ? 64u : a.cout <= 128 ? 128u : 256u;
    const uint32_t ncols = 2u * ncols1;

    if (tid == 0) {
        for (int s = 0; s < stages; ++s) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], 1);
        }
        mbar_init(&accf[0], 1);
        mbar_init(&accf[1], 1);
        mbar_init(&acce[0], kEpiThreads);
        mbar_init(&acce[1], kEpiThreads);
        mbar_init(fin, 1);
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
    grid_dep_wait();
    const uint32_t tmem = *tslot;

    if (warp == 0) {
        if (lane == 0) {   // producer
            int kg = 0;
            for (int t = blockIdx.x; t < ntiles && !*abort_flag; t += gridDim.x) {
                int x0, y0, img;
                tile_origin(t, tiles_x, tiles_y, x0, y0, img);
                for (int k = 0; k < nk; ++k, ++kg) {
                    const int s = kg % stages;
                    const uint32_t use = (uint32_t)(kg / stages);
                    if (use > 0 && !mbar_wait_bounded(&empty[s], (use - 1u) & 1u, a.err)) {
                        *abort_flag = 1;
                        break;
                    }
                    uint8_t* sa = smem + s * stage_bytes;
                    mbar_expect_tx(&full[s], (uint32_t)(a_bytes + nb * b_bytes));
                    if (rows) {
                        const int dx = k / kc, c = k - dx * kc;
                        tma_load_4d(sa, &mx, c * 32, x0 + dx - 1, y0 - 1, img, &full[s]);
                        for (int dy = 0; dy < 3; ++dy)
                            tma_load_2d(sa + a_bytes + dy * b_bytes, &mw, (dy * 3 + dx) * a.cin + c * 32, 0, &full[s]);
                    } else {
                        const int tap = k / kc, c = k - tap * kc;
                        tma_load_4d(sa, &mx, c * 32, x0 + tap % 3 - 1, y0 + tap / 3 - 1, img, &full[s]);
                        tma_load_2d(sa + a_bytes, &mw, tap * a.cin + c * 32, 0, &full[s]);
                    }
                }
            }
        }
    } else if (warp == 1) {
        if (lane == 0) {   // MMA issuer
            const uint32_t idesc = umma_idesc_bf16(128u, (uint32_t)a.cout);
            const int b_step = b_bytes >> 4;   // one weight box in 16-byte units
            int kg = 0, i = 0;
            bool ok = true;
            for (int t = blockIdx.x; t < ntiles && ok; t += gridDim.x, ++i) {
                const int acc = i & 1;
                const uint32_t use = (uint32_t)(i >> 1);
                if (use > 0 && !mbar_wait_bounded(&acce[acc], (use - 1u) & 1u, a.err)) {
                    *abort_flag = 1;
                    break;
                }
                tc_fence_after();
                const uint32_t d = tmem + (uint32_t)acc * ncols1;
                for (int k = 0; k < nk; ++k, ++kg) {
                    const int s = kg % stages;
                    if (!mbar_wait_bounded(&full[s], (uint32_t)(kg / stages) & 1u, a.err)) {
                        *abort_flag = 1;
                        ok = false;
                        break;
                    }
                    tc_fence_after();
                    const uint32_t sa = smem_u32(smem + s * stage_bytes);
                    // start fields (16-byte units) stay below 2^14: shared memory < 256 KB
                    const uint64_t a0 = umma_desc_sw64(sa), b0 = umma_desc_sw64(sa + (uint32_t)a_bytes);
#pragma unroll
                    for (int dy = 0; dy < nb; ++dy) {
                        const uint64_t ta = a0 + (uint64_t)(dy * kTileX * 4), tb = b0 + (uint64_t)(dy * b_step);
                        umma_bf16(d, ta, tb, idesc, (k | dy) != 0 ? 1u : 0u);
                        umma_bf16(d, ta + 2u, tb + 2u, idesc, 1u);
                    }
                    umma_commit(&empty[s]);
                }
                if (ok) umma_commit(&accf[acc]);
            }
            umma_commit(fin);
            mbar_wait_bounded(fin, 0u, a.err);   // nothing may be in flight when TMEM is freed
        }
    } else {
        // epilogue: warp w reads TMEM lanes 32 (w % 4) .. +31, the tile's pixels of that quarter
        const int q = warp & 3;
        const int p = q * 32 + lane;
        int i = 0;
        for (int t = blockIdx.x; t < ntiles; t += gridDim.x, ++i) {
            const int acc = i & 1;
            const bool ready = mbar_wait_bounded(&accf[acc], (uint32_t)(i >> 1) & 1u, a.err);
            __syncwarp();
            tc_fence_after();
            if (!__all_sync(0xFFFFFFFFu, ready) || *abort_flag) break;
            int x0, y0, img;
            tile_origin(t, tiles_x, tiles_y, x0, y0, img);
            const int y = y0 + p / kTileX, x = x0 + p % kTileX;
            const bool inside = y < a.H && x < a.W;
            const size_t pix = ((size_t)img * a.H + y) * a.W + x;
            const uint32_t base = tmem + (uint32_t)acc * ncols1 + ((uint32_t)(q * 32) << 16);
            const EpiDst dst = epi_dst(a, img, x, y, inside, 16);   // y-neighbour: lane ^ 16 (16-pixel rows)
            for (int c0 = 0; c0 < a.cout; c0 += 16) {
                uint32_t r[16];
                tmem_ld16(base + (uint32_t)c0, r);
                tmem_ld_wait();
                float v[16];
#pragma unroll
                for (int j = 0; j < 16; ++j) v[j] = __uint_as_float(r[j]);
                add_bias16(a.bias, c0, v);
                if (a.add_par && inside) add_parity(a, v, pix_add(a, img, x, y), c0);
#pragma unroll
                for (int j = 0; j < 16; ++j)
                    if (a.flags & kConvRelu) v[j] = fmaxf(v[j], 0.0f);
                if (a.flags & kConvF32Out) {
                    if (!inside) continue;
                    store_f32(reinterpret_cast<float*>(a.out) + pix * a.out_c + a.out_off + c0, v,
                              min(16, a.n_store - c0));
                } else {
                    epilogue_bf16(a, v, dst, c0, 16, ebuf + 64 * q);
                }
            }
            tc_fence_before();
            mbar_arrive(&acce[acc]);
        }
    }
    __syncthreads();
    if (warp == 1) tmem_dealloc(tmem, ncols);
}

// ---------------------------------------------------------------------------------------------
// Halo tiles: outputs of up to 32 channels whose weights fit in shared memory (the
// full-resolution layers). Tiles of 8 x 16 pixels (x by y, M = 128). The CTA loads all weights
// once ({32 Cin, Cout} boxes per tap and input chunk, 64-byte swizzled) and keeps them; per
// 32-channel input chunk a stage holds the chunk's 10 x 18-pixel halo box (180 pixel rows), so
// that the A operand of tap (dy, dx) is that box at start offset (10 dy + dx) rows, 8-row groups
// (one tile row) 10 rows apart. Each input chunk is read once per tile (with its halo, 1.4x),
// and no weights per tile. Two layouts of the box, chosen by the input's pixel stride:
//  * rows (rb = 64, or 32 for an input of 16 channels), when the chunk is the whole pixel: one
//    TMA box of rb-byte pixel rows in the K-major layout with rb-byte swizzle. The tensor core
//    applies the swizzle on the absolute shared-memory address bits, as the TMA does when it
//    writes the box, so an operand may start at any row of it (descriptor base offset 0).
//  * planes (rb = 16), when the chunk is part of a wider pixel: four 8-channel planes without
//    swizzle (180 rows of 16 bytes each, planes 2944 bytes apart: a TMA destination must be
//    128-byte aligned), core matrices of 8 pixels 160 bytes apart, K halves one plane pair apart.
// Measured on the 1080p denoiser layers (ncu, cold): 32 -> 32 layers 110 -> 95 us with rows;
// the 96-channel input (192-byte pixels read 64 bytes at a time) 211 us with planes, 281 with
// rows; the 16-channel input 111 -> 85 us (rows of 32 bytes: half the MMAs).

constexpr int kHaloX = 8, kHaloY = 16;
constexpr int kHaloBoxX = kHaloX + 2, kHaloBoxY = kHaloY + 2;
constexpr int kHaloRows = kHaloBoxX * kHaloBoxY;                   // 180 pixel rows
constexpr int kHaloPlane = kHaloRows * 16;                         // 8 channels: 2880 bytes
constexpr int kHaloPlaneStride = (kHaloPlane + 127) & ~127;        // 2944
constexpr int kHaloStage = (4 * kHaloPlaneStride + 1023) & ~1023;  // 12288 (>= 180 x 64): 1024-byte aligned
constexpr int kHaloStages = 4;
constexpr int kHaloWeightMax = 96 * 1024;

// kRb: 16 (planes), 32 or 64 (rows of that many bytes). The MMA issuer's loop over the nine taps
// is unrolled with the operand offsets as constants added to the descriptors' start fields: with
// up to 54 MMAs per tile a single issuing thread must not fall behind the tensor core.
template <int kRb>
__global__ void __launch_bounds__(kConvThreads) k_conv3x3_halo(const __grid_constant__ CUtensorMap mx,
                                                               const __grid_constant__ CUtensorMap mw, ConvArgs a,
                                                               int tiles_x, int tiles_y, int ntiles) {
    constexpr int rb = kRb;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    const int kc = a.cin / 32;
    const int b_bytes = a.cout * 64;   // one weight box: a multiple of 1024 bytes
    const int w_bytes = 9 * kc * b_bytes;
    uint8_t* wsm = smem;               // box (chunk c, tap) at (9 c + tap) * b_bytes
    uint8_t* stage0 = smem + w_bytes;
    uint64_t* full = reinterpret_cast<uint64_t*>(stage0 + kHaloStages * kHaloStage);
    uint64_t* empty = full + kHaloStages;
    uint64_t* wbar = empty + kHaloStages;
    uint64_t* accf = wbar + 1;
    uint64_t* acce = accf + 2;
    uint64_t* fin = acce + 2;
    uint32_t* tslot = reinterpret_cast<uint32_t*>(fin + 1);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tslot + 1);
    uint4* ebuf = reinterpret_cast<uint4*>((reinterpret_cast<uintptr_t>(tslot + 2) + 15) & ~(uintptr_t)15);

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t ncols1 = a.cout <= 32 ? 32u : 64u;
    const uint32_t ncols = 2u * ncols1;

    if (tid == 0) {
        for (int s = 0; s < kHaloStages; ++s) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], 1);
        }
        mbar_init(wbar, 1);
        mbar_init(&accf[0], 1);
        mbar_init(&accf[1], 1);
        mbar_init(&acce[0], kEpiThreads);
        mbar_init(&acce[1], kEpiThreads);
        mbar_init(fin, 1);
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
    grid_dep_wait();
    const uint32_t tmem = *tslot;

    if (warp == 0) {
        if (lane == 0) {   // producer: the weights once, then one halo box per tile and chunk
            mbar_expect_tx(wbar, (uint32_t)w_bytes);
            for (int c = 0; c < kc; ++c)
                for (int tap = 0; tap < 9; ++tap)
                    tma_load_2d(wsm + (9 * c + tap) * b_bytes, &mw, tap * a.cin + c * 32, 0, wbar);
            int kg = 0;
            for (int t = blockIdx.x; t < ntiles && !*abort_flag; t += gridDim.x) {
                const int per_img = tiles_x * tiles_y, img = t / per_img, r = t - img * per_img;
                const int y0 = (r / tiles_x) * kHaloY, x0 = (r % tiles_x) * kHaloX;
                for (int c = 0; c < kc; ++c, ++kg) {
                    const int s = kg % kHaloStages;
                    const uint32_t use = (uint32_t)(kg / kHaloStages);
                    if (use > 0 && !mbar_wait_bounded(&empty[s], (use - 1u) & 1u, a.err)) {
                        *abort_flag = 1;
                        break;
                    }
                    uint8_t* sa = stage0 + s * kHaloStage;
                    if (smem_u32(sa) & 1023u) {   // stages start 1024-byte aligned (weights: 1024-byte boxes)
                        // (planes then start 128-byte aligned)
                        atomicOr(a.err, kErrTmaWait);
                        *abort_flag = 1;
                        break;
                    }
                    if (kRb == 16) {
                        mbar_expect_tx(&full[s], (uint32_t)(4 * kHaloPlane));
                        for (int j = 0; j < 4; ++j)
                            tma_load_4d(sa + j * kHaloPlaneStride, &mx, c * 32 + j * 8, x0 - 1, y0 - 1, img,
                                        &full[s]);
                    } else {
                        mbar_expect_tx(&full[s], (uint32_t)(kHaloRows * rb));
                        tma_load_4d(sa, &mx, c * 32, x0 - 1, y0 - 1, img, &full[s]);
                    }
                }
            }
        }
    } else if (warp == 1) {
        if (lane == 0) {   // MMA issuer
            const uint32_t idesc = umma_idesc_bf16(128u, (uint32_t)a.cout);
            bool ok = mbar_wait_bounded(wbar, 0u, a.err);
            if (!ok) *abort_flag = 1;
            tc_fence_after();
            const uint32_t wb0 = smem_u32(wsm);
            const int b_step = b_bytes >> 4;   // one tap's weight box in 16-byte units
            int kg = 0, i = 0;
            for (int t = blockIdx.x; t < ntiles && ok; t += gridDim.x, ++i) {
                const int acc = i & 1;
                const uint32_t use = (uint32_t)(i >> 1);
                if (use > 0 && !mbar_wait_bounded(&acce[acc], (use - 1u) & 1u, a.err)) {
                    *abort_flag = 1;
                    break;
                }
                tc_fence_after();
                const uint32_t d = tmem + (uint32_t)acc * ncols1;
                for (int c = 0; c < kc; ++c, ++kg) {
                    const int s = kg % kHaloStages;
                    if (!mbar_wait_bounded(&full[s], (uint32_t)(kg / kHaloStages) & 1u, a.err)) {
                        *abort_flag = 1;
                        ok = false;
                        break;
                    }
                    tc_fence_after();
                    const uint32_t sa = smem_u32(stage0 + s * kHaloStage);
                    // descriptors of the tap-(0, 0) operands; a tap adds its offset (16-byte
                    // units) to the start field, which stays below 2^14 (shared memory < 256 KB)
                    const uint64_t a0 = kRb == 16 ? umma_desc_dense(sa, (uint32_t)kHaloPlaneStride, kHaloBoxX * 16u)
                                                  : umma_desc_swz(sa, (uint32_t)kRb, (uint32_t)(kHaloBoxX * kRb));
                    const uint64_t b0 = umma_desc_sw64(wb0 + (uint32_t)(9 * c * b_bytes));
                    constexpr int nkk = kRb == 32 ? 1 : 2;
#pragma unroll
                    for (int tap = 0; tap < 9; ++tap) {
                        const int off = ((tap / 3) * kHaloBoxX + tap % 3) * kRb;
#pragma unroll
                        for (int kk = 0; kk < nkk; ++kk) {
                            const int aoff = kRb == 16 ? 2 * kk * kHaloPlaneStride + off : off + kk * 32;
                            umma_bf16(d, a0 + (uint64_t)(aoff >> 4), b0 + (uint64_t)(tap * b_step + kk * 2), idesc,
                                      (c | tap | kk) != 0 ? 1u : 0u);
                        }
                    }
                    umma_commit(&empty[s]);
                }
                if (ok) umma_commit(&accf[acc]);
            }
            umma_commit(fin);
            mbar_wait_bounded(fin, 0u, a.err);   // nothing may be in flight when TMEM is freed
        }
    } else {
        const int q = warp & 3;
        const int p = q * 32 + lane;
        int i = 0;
        for (int t = blockIdx.x; t < ntiles; t += gridDim.x, ++i) {
            const int acc = i & 1;
            const bool ready = mbar_wait_bounded(&accf[acc], (uint32_t)(i >> 1) & 1u, a.err);
            __syncwarp();
            tc_fence_after();
            if (!__all_sync(0xFFFFFFFFu, ready) || *abort_flag) break;
            const int per_img = tiles_x * tiles_y, img = t / per_img, r = t - img * per_img;
            const int y = (r / tiles_x) * kHaloY + p / kHaloX, x = (r % tiles_x) * kHaloX + p % kHaloX;
            const bool inside = y < a.H && x < a.W;
            const size_t pix = ((size_t)img * a.H + y) * a.W + x;
            const uint32_t base = tmem + (uint32_t)acc * ncols1 + ((uint32_t)(q * 32) << 16);
            const EpiDst dst = epi_dst(a, img, x, y, inside, 8);   // y-neighbour: lane ^ 8 (8-pixel rows)
            for (int c0 = 0; c0 < a.cout; c0 += 16) {
                uint32_t rr[16];
                tmem_ld16(base + (uint32_t)c0, rr);
                tmem_ld_wait();
                float v[16];
#pragma unroll
                for (int j = 0; j < 16; ++j) v[j] = __uint_as_float(rr[j]);
                add_bias16(a.bias, c0, v);
                if (a.add_par && inside) add_parity(a, v, pix_add(a, img, x, y), c0);
#pragma unroll
                for (int j = 0; j < 16; ++j)
                    if (a.flags & kConvRelu) v[j] = fmaxf(v[j], 0.0f);
                if (a.flags & kConvF32Out) {
                    if (!inside) continue;
                    store_f32(reinterpret_cast<float*>(a.out) + pix * a.out_c + a.out_off + c0, v,
                              min(16, a.n_store - c0));
                } else {
                    epilogue_bf16(a, v, dst, c0, 8, ebuf + 64 * q);
                }
            }
            tc_fence_before();
            mbar_arrive(&acce[acc]);
        }
    }
    __syncthreads();
    if (warp == 1) tmem_dealloc(tmem, ncols);
}

// ---------------------------------------------------------------------------------------------
// Row tiles: a CTA keeps the weights of its output channels in shared memory for all its tiles of 128 x
// kR pixels, whose kR rows of accumulators lie next to each other in TMEM. M = 128 pixels of one input
// row; that row against the weights of its vertical taps is one MMA of N = up to 3 Cout, which adds to
// the accumulators of the rows r - 1, r and r + 1: the A operand, whose shared-memory reads bound MMAs
// of small N (128 rows of 32 bytes take 32 cycles; N = 32 alone 16), is shared by the taps.
//   stages    the tile's kR + 2 input rows of 130 pixels x 32 channels in one box (64-byte swizzle; 32
//             for a 16-channel input); the horizontal taps are its windows from pixel 0, 1 and 2.
//   order     FP32 sums are taken as the other kernels take them: (chunk, dy, dx), or with kDxOuter (dx,
//             chunk, dy), for which a tile's chunks all stay in shared memory.
//   issue     a warp's MMAs follow one another only as fast as it issues them (a wait on a barrier costs
//             about 115 cycles, a commit 36, a dependent instruction 5), so a tile's MMAs are unrolled
//             with their offsets as constants, a tile has one barrier per chunk for its loads, one for
//             its sums and one for their release, and two warps issue, for every other tile each: while
//             one waits or computes addresses, the other's MMAs run.
//   epilogue  up to four groups of four warps take the rows in turn, kG columns at a time: bias, addend,
//             ReLU, and through swizzled shared memory out by TMA (the tensor map clips the edges; the
//             nearest upsampling is four more stores of the same bytes). kMode is a template parameter
//             because the pooled rows and the addend of a general one lived in local memory: 540
//             instructions per 32 columns instead of 200, and twice the time of the whole kernel.
// What bounds it: DRAM at full resolution, the operand reads of shared memory otherwise. Before and after,
// cold: 32 -> 32 channels on 1080p 72 -> 48 us, 32 -> 4 (FP32) 60 -> 44; on 540 x 960 32 -> 64 44 -> 27,
// 64 -> 64 55 -> 37, 64 -> 128 88 -> 58; 64 -> 64 on 539 x 963 66 -> 36.
constexpr int kRowGroups = 4;
constexpr int kRowThreads = 96 + kRowGroups * kEpiThreads;   // producer, issuer, epilogue, issuer
constexpr int kRowMaxStages = 8;
constexpr int kRowMaxSets = 8;
constexpr int kRowMaxChunks = 8;
constexpr int kRowPix = 130;

struct RowPlan {
    int nxs, nyb;        // tiles per image row and column
    int items;           // tiles
    int ring, sets;      // input boxes of each issuer; tiles whose accumulators TMEM holds
    int groups;          // epilogue groups at work
};

__device__ __forceinline__ void tma_store_4d(const CUtensorMap* map, const void* src, int c0, int c1, int c2, int c3) {
    asm volatile("cp.async.bulk.tensor.4d.global.shared::cta.bulk_group [%0, {%1, %2, %3, %4}], [%5];" ::"l"(
                     reinterpret_cast<uint64_t>(map)),
                 "r"(c0), "r"(c1), "r"(c2), "r"(c3), "r"(smem_u32(src))
                 : "memory");
}
__device__ __forceinline__ void tma_store_5d(const CUtensorMap* map, const void* src, int c0, int c1, int c2, int c3,
                                             int c4) {
    asm volatile("cp.async.bulk.tensor.5d.global.shared::cta.bulk_group [%0, {%1, %2, %3, %4, %5}], [%6];" ::"l"(
                     reinterpret_cast<uint64_t>(map)),
                 "r"(c0), "r"(c1), "r"(c2), "r"(c3), "r"(c4), "r"(smem_u32(src))
                 : "memory");
}
__device__ __forceinline__ void tma_store_commit() { asm volatile("cp.async.bulk.commit_group;" ::: "memory"); }
template <int kPending>
__device__ __forceinline__ void tma_store_wait_read() {   // at most kPending groups still read shared memory
    asm volatile("cp.async.bulk.wait_group.read %0;" ::"n"(kPending) : "memory");
}
__device__ __forceinline__ void tma_store_wait_all() { asm volatile("cp.async.bulk.wait_group 0;" ::: "memory"); }
__device__ __forceinline__ void fence_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

__device__ __forceinline__ uint32_t relu2(uint32_t v) {
    __nv_bfloat162 h = *reinterpret_cast<__nv_bfloat162*>(&v);
    h = __hmax2(h, __nv_bfloat162{__nv_bfloat16_raw{0}, __nv_bfloat16_raw{0}});
    return *reinterpret_cast<uint32_t*>(&h);
}
__host__ __device__ constexpr int row_stage_bytes(int rb, int r) {
    return ((r + 2) * kRowPix * rb + 511) & ~511;
}

// The 2 x 2 average of two rows' 32 (kG) stored channels of a warp's pixels: the lanes of a pixel pair
// swap halves of their channels, and each averages its half, (((0 + v(x, y)) + v(x + 1, y)) +
// v(x, y + 1)) + v(x + 1, y + 1) times 1/4 rounded to bf16, and stores it.
template <int kG>
__device__ __forceinline__ void pool_store(const uint32_t (&r0)[kG / 2], const uint32_t (&r1)[kG / 2], bool inside,
                                           __nv_bfloat16* dst) {
    constexpr int kH = kG / 4;   // registers (two channels each) of half the channels
    const bool odd = (threadIdx.x & 1) != 0;
    uint32_t o[kH];
#pragma unroll
    for (int j = 0; j < kH; ++j) {
        const uint32_t own0 = odd ? r0[kH + j] : r0[j], own1 = odd ? r1[kH + j] : r1[j];
        const uint32_t got0 = __shfl_xor_sync(0xFFFFFFFFu, odd ? r0[j] : r0[kH + j], 1);
        const uint32_t got1 = __shfl_xor_sync(0xFFFFFFFFu, odd ? r1[j] : r1[kH + j], 1);
        const uint32_t a = odd ? got0 : own0, b = odd ? own0 : got0, c = odd ? got1 : own1, d = odd ? own1 : got1;
        float lo = 0.0f + __uint_as_float(a << 16), hi = 0.0f + __uint_as_float(a & 0xFFFF0000u);
        lo = lo + __uint_as_float(b << 16);
        hi = hi + __uint_as_float(b & 0xFFFF0000u);
        lo = lo + __uint_as_float(c << 16);
        hi = hi + __uint_as_float(c & 0xFFFF0000u);
        lo = lo + __uint_as_float(d << 16);
        hi = hi + __uint_as_float(d & 0xFFFF0000u);
        o[j] = pack_bf16x2(lo * 0.25f, hi * 0.25f);
    }
    if (!inside) return;
#pragma unroll
    for (int j = 0; j < kH; j += 4)
        reinterpret_cast<uint4*>(dst + (odd ? kG / 2 : 0))[j / 4] = make_uint4(o[j], o[j + 1], o[j + 2], o[j + 3]);
}

// kMode: what the epilogue does besides bias, ReLU and the store
enum RowMode { kRowPlain = 0, kRowPool = 1, kRowAdd = 2, kRowF32 = 3 };
template <int kRb, int kG, int kR, bool kDxOuter, int kMode>
__global__ void __launch_bounds__(kRowThreads, 1) k_conv_rows(const __grid_constant__ CUtensorMap mx,
                                                              const __grid_constant__ CUtensorMap mw,
                                                              const __grid_constant__ CUtensorMap mo,
                                                              const __grid_constant__ CUtensorMap mu, ConvArgs a,
                                                              RowPlan p) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    constexpr int kStage = row_stage_bytes(kRb, kR);
    const int kc = a.cin / 32, nco = a.cout;
    const int b_bytes = nco * 64;   // one tap's weight box
    uint8_t* wsm = smem;              // box (chunk c, dx, dy) at ((3 c + dx) 3 + 2 - dy) b_bytes
    uint8_t* stage0 = wsm + 9 * kc * b_bytes;
    uint8_t* stores = stage0 + 2 * p.ring * kStage;   // 64 kG bytes per epilogue warp
    float* bsm = reinterpret_cast<float*>(stores + p.groups * 4 * 64 * kG);   // the bias
    uint64_t* full = reinterpret_cast<uint64_t*>(bsm + 128);
    uint64_t* empty = full + kRowMaxStages;
    uint64_t* sfull = empty + kRowMaxStages;   // a set's sums are complete
    uint64_t* sempty = sfull + kRowMaxSets;    // and have been read
    uint64_t* wbar = sempty + kRowMaxSets;     // weight boxes of (chunk, dx)
    uint64_t* fin = wbar + 3 * kRowMaxChunks;
    uint32_t* tslot = reinterpret_cast<uint32_t*>(fin + 1);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tslot + 1);

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    if (tid == 0) {
        for (int s = 0; s < 2 * p.ring; ++s) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], 1);
        }
        for (int i = 0; i < p.sets; ++i) {
            mbar_init(&sfull[i], 1);
            mbar_init(&sempty[i], 4 * kR);
        }
        for (int i = 0; i < 3 * kc; ++i) mbar_init(&wbar[i], 1);
        mbar_init(fin, 2);
        *abort_flag = 0;
        mbar_fence_init();
    }
    if (warp == 1) {
        tmem_alloc(tslot, 512u);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    grid_dep_launch();
    grid_dep_wait();
    // -0 adds nothing, not even to a -0
    for (int i = tid; i < nco; i += blockDim.x) bsm[i] = a.bias ? __ldg(a.bias + i) : -0.0f;
    __syncthreads();
    const uint32_t tmem = *tslot;
    const int per_img = p.nxs * p.nyb;

    if (warp == 0) {
        if (lane == 0) {   // producer: the weights in the order of their use, then the tiles' rows
            for (int i = 0; i < 3 * kc; ++i) {
                const int c = kDxOuter ? i % kc : i / 3, dx = kDxOuter ? i / kc : i % 3, wi = 3 * c + dx;
                mbar_expect_tx(&wbar[wi], (uint32_t)(3 * b_bytes));
                for (int dy = 0; dy < 3; ++dy)
                    tma_load_2d(wsm + (3 * wi + 2 - dy) * b_bytes, &mw, (3 * dy + dx) * a.cin + 32 * c, 0, &wbar[wi]);
            }
            // Each issuer has a ring of its own, so that whoever waits for a stage's next load has waited
            // for its last one (a barrier tells phases apart by parity alone).
            int pos = 0, other = 0;   // the next stage of this tile's ring, and of the other one
            uint32_t use = 0, other_use = 0;
            int base = 0;
            bool ok = true;
            for (int t = blockIdx.x; t < p.items && ok; t += gridDim.x) {
                const int img = t / per_img, r = t - img * per_img, yb = r / p.nxs;
                const int x = (r - yb * p.nxs) * 128 - 1, y = yb * kR - 1;
                for (int c = 0; c < kc; ++c) {
                    const int s = base + pos;
                    if (use > 0) ok = mbar_wait_bounded(&empty[s], (use - 1u) & 1u, a.err);
                    if (!ok || *abort_flag) {
                        *abort_flag = 1;
                        ok = false;
                        break;
                    }
                    mbar_expect_tx(&full[s], (uint32_t)((kR + 2) * kRowPix * kRb));
                    tma_load_4d(stage0 + s * kStage, &mx, 32 * c, x, y, img, &full[s]);
                    if (++pos == p.ring) {
                        pos = 0;
                        ++use;
                    }
                }
                if (!ok) break;
                const int pt = pos;
                pos = other;
                other = pt;
                const uint32_t ut = use;
                use = other_use;
                other_use = ut;
                base = p.ring - base;
            }
            // no load may be in flight when the CTA ends, whoever gave up
            for (int w = 0; w < 2; ++w) {
                for (int i = 0; i < p.ring; ++i) {
                    const uint32_t uses = use + (i < pos ? 1u : 0u);
                    if (uses > 0) mbar_wait_bounded(&full[base + i], (uses - 1u) & 1u, a.err);
                }
                pos = other;
                use = other_use;
                base = p.ring - base;
            }
            for (int i = 0; i < 3 * kc; ++i) mbar_wait_bounded(&wbar[i], 0u, a.err);
        }
    } else if (warp == 1 || warp == 2 + 4 * p.groups) {
        // two MMA issuers take the tiles in turn; the whole warp walks them, so that what an MMA needs is
        // warp-uniform, and one elected lane issues
        constexpr uint32_t kHi = (8u * kRb >> 4) | (1u << 14) | ((kRb == 64 ? 4u : 6u) << 29);   // umma_desc_swz
        constexpr uint32_t kHiB = (512u >> 4) | (1u << 14) | (4u << 29);                         // umma_desc_sw64
        constexpr uint32_t kRow = kRowPix * kRb / 16, kPixel = kRb / 16;                         // of a box
        constexpr int nkk = kRb / 32;
        const bool leader = elect_one();
        const uint32_t nfield = (uint32_t)(nco >> 3) << 17, id1 = umma_idesc_bf16(128u, 0u) + nfield;
        const uint32_t ids[3] = {id1, id1 + nfield, id1 + 2u * nfield};
        const uint32_t wlo = (smem_u32(wsm) >> 4) | (1u << 16), slo = (smem_u32(stage0) >> 4) | (1u << 16);
        const uint32_t bstep = (uint32_t)b_bytes >> 4;
        const int who = warp == 1 ? 0 : 1;
        int s0 = 0, set = 0, kt = who;   // the tile's first stage and its set
        uint32_t use0 = 0, phase = 0;
        bool ok = true;
        const uint32_t sring = slo + (uint32_t)(who * p.ring * (kStage >> 4));
        full += who * p.ring;
        empty += who * p.ring;
        auto next_set = [&](int n) {
            set += n;
            while (set >= p.sets) {
                set -= p.sets;
                phase ^= 1u;
            }
        };
        next_set(who);
        // all MMAs of input row rr at horizontal taps dx0 .. dx1 - 1 (a: the stage, b: the first tap's
        // boxes); fresh: row rr of the accumulators gets its first products
        auto mma_row = [&](uint32_t dt, uint32_t ar, uint32_t b, int rr, int dx0, int dx1, bool fresh) {
            const int lo = rr < 2 ? 0 : rr - 2, n = (rr < kR ? rr : kR - 1) - lo + 1;   // rows lo ..: tap dy = rr - o
            const uint32_t d = dt + (uint32_t)(lo * nco);
#pragma unroll
            for (int dx = dx0; dx < dx1; ++dx)
#pragma unroll
                for (int kk = 0; kk < nkk; ++kk) {
                    const uint32_t al = ar + (uint32_t)dx * kPixel + 2u * (uint32_t)kk;
                    const uint32_t bx = b + (uint32_t)(3 * (dx - dx0)) * bstep + 2u * (uint32_t)kk;
                    const uint32_t bo = bx + (uint32_t)(2 - rr + lo) * bstep;
                    if (dx == dx0 && kk == 0 && rr < kR && fresh) {
                        if (rr > 0) umma_bf16_lo(d, al, kHi, bo, kHiB, ids[n - 2 < 0 ? 0 : n - 2], 1u);
                        umma_bf16_lo(dt + (uint32_t)(rr * nco), al, kHi, bx + 2u * bstep, kHiB, id1, 0u);
                    } else {
                        umma_bf16_lo(d, al, kHi, bo, kHiB, ids[n - 1], 1u);
                    }
                }
        };
        for (int t = blockIdx.x + who * gridDim.x; t < p.items && ok; t += 2 * gridDim.x, kt += 2) {
            const uint32_t dt = tmem + (uint32_t)(set * kR * nco);
            if (kt >= p.sets) ok = mbar_wait_bounded(&sempty[set], phase ^ 1u, a.err);
            ok = __all_sync(0xFFFFFFFFu, ok);
            if (kDxOuter) {
#pragma unroll
                for (int dx = 0; dx < 3; ++dx) {
                    int s = s0;
                    uint32_t use = use0;
                    for (int c = 0; c < kc && ok; ++c) {
                        const int wi = 3 * c + dx;
                        if (kt < 2) ok = __all_sync(0xFFFFFFFFu, mbar_wait_bounded(&wbar[wi], 0u, a.err));
                        if (dx == 0) ok = __all_sync(0xFFFFFFFFu, mbar_wait_bounded(&full[s], use & 1u, a.err) && ok);
                        if (!ok) break;
                        tc_fence_after();
                        if (leader) {
                            const uint32_t b = wlo + (uint32_t)(3 * wi) * bstep;
                            const uint32_t as = sring + (uint32_t)s * (uint32_t)(kStage >> 4);
                            if (dx == 0 && c == 0) {
#pragma unroll
                                for (int rr = 0; rr < kR + 2; ++rr)
                                    mma_row(dt, as + (uint32_t)rr * kRow, b, rr, dx, dx + 1, true);
                            } else {
#pragma unroll
                                for (int rr = 0; rr < kR + 2; ++rr)
                                    mma_row(dt, as + (uint32_t)rr * kRow, b, rr, dx, dx + 1, false);
                            }
                            if (dx == 2) umma_commit(&empty[s]);
                        }
                        __syncwarp();
                        if (++s == p.ring) {
                            s = 0;
                            ++use;
                        }
                    }
                }
            } else {
                int s = s0;
                uint32_t use = use0;
                for (int c = 0; c < kc && ok; ++c) {
                    if (kt < 2) {
                        for (int dx = 0; dx < 3; ++dx) ok = mbar_wait_bounded(&wbar[3 * c + dx], 0u, a.err) && ok;
                    }
                    ok = __all_sync(0xFFFFFFFFu, mbar_wait_bounded(&full[s], use & 1u, a.err) && ok);
                    if (!ok) break;
                    tc_fence_after();
                    if (leader) {
                        const uint32_t b = wlo + (uint32_t)(9 * c) * bstep;
                        const uint32_t as = sring + (uint32_t)s * (uint32_t)(kStage >> 4);
                        if (c == 0) {
#pragma unroll
                            for (int rr = 0; rr < kR + 2; ++rr) mma_row(dt, as + (uint32_t)rr * kRow, b, rr, 0, 3, true);
                        } else {
#pragma unroll
                            for (int rr = 0; rr < kR + 2; ++rr) mma_row(dt, as + (uint32_t)rr * kRow, b, rr, 0, 3, false);
                        }
                        umma_commit(&empty[s]);
                    }
                    __syncwarp();
                    if (++s == p.ring) {
                        s = 0;
                        ++use;
                    }
                }
            }
            if (!ok) break;
            if (leader) umma_commit(&sfull[set]);
            __syncwarp();
            s0 += kc;
            while (s0 >= p.ring) {
                s0 -= p.ring;
                ++use0;
            }
            next_set(2);
        }
        if (!ok) *abort_flag = 1;
        if (leader) {
            umma_commit(fin);
            mbar_wait_bounded(fin, 0u, a.err);   // nothing may be in flight when TMEM is freed
        }
        __syncwarp();
    } else {
        const int q = warp & 3, group = (warp - 2) >> 2;
        uint8_t* sbuf = stores + (warp - 2) * 64 * kG;
        const uint32_t lane0 = tmem + ((uint32_t)(q * 32) << 16);
        const bool relu = (a.flags & kConvRelu) != 0, leader = elect_one();
        constexpr int kUnit = kMode == kRowPool ? 2 : 1;   // rows taken together
        const int sw = kG == 32 ? (lane >> 1) & 3 : (lane >> 2) & 1;
        uint4* sb = reinterpret_cast<uint4*>(sbuf) + lane * (kG / 8);
        int set = 0, turn = 0;
        uint32_t phase = 0;
        bool ok = true;
        for (int t = blockIdx.x; t < p.items && ok; t += gridDim.x) {
            const int img = t / per_img, rt = t - img * per_img, yb = rt / p.nxs;
            const int x0 = (rt - yb * p.nxs) * 128 + q * 32, x = x0 + lane;
#pragma unroll 1
            for (int o0 = 0; o0 < kR; o0 += kUnit) {
                const bool mine = turn == group;
                if (++turn == p.groups) turn = 0;
                if (!mine) continue;
                // the addend, in flight while the tile's sums are awaited (one column group): kG / 8 lanes to
                // a pixel, whole sectors each; every lane gets its own pixel's through the store buffer
                constexpr int kParts = kG / 8;
                uint4 add[kMode == kRowAdd ? kParts : 1];
                if (kMode == kRowAdd) {
                    const int y = yb * kR + o0;
#pragma unroll
                    for (int j = 0; j < kParts; ++j) {
                        const int xa = x0 + j * (32 / kParts) + lane / kParts;
                        const bool in = xa < a.W && y < a.H;
                        add[j] = in ? __ldg(reinterpret_cast<const uint4*>(
                                                reinterpret_cast<const __nv_bfloat16*>(a.add_par) +
                                                pix_add(a, img, xa, y)) + lane % kParts)
                                    : make_uint4(0u, 0u, 0u, 0u);
                    }
                }
                ok = mbar_wait_bounded(&sfull[set], phase, a.err) && !*abort_flag;
                ok = __all_sync(0xFFFFFFFFu, ok);
                if (!ok) break;
                tc_fence_after();
#pragma unroll 1
                for (int c0 = 0; c0 < nco; c0 += kG) {
                    uint32_t pk[kUnit][kG / 2];   // the rows' stored values
#pragma unroll
                    for (int u = 0; u < kUnit; ++u) {
                        const int o = o0 + u, y = yb * kR + o;
                        uint32_t r[kG];
                        const uint32_t col = lane0 + (uint32_t)((set * kR + o) * nco + c0);
                        if constexpr (kG == 32) tmem_ld32(col, r);
                        else tmem_ld16(col, r);
                        tmem_ld_wait();
                        if (c0 + kG >= nco) {
                            tc_fence_before();
                            __syncwarp();
                            if (leader) mbar_arrive(&sempty[set]);
                        }
                        float v[kG];
                        const float4* b4 = reinterpret_cast<const float4*>(bsm + c0);
#pragma unroll
                        for (int j = 0; j < kG; j += 4) {
                            const float4 b = b4[j / 4];
                            v[j] = __uint_as_float(r[j]) + b.x;
                            v[j + 1] = __uint_as_float(r[j + 1]) + b.y;
                            v[j + 2] = __uint_as_float(r[j + 2]) + b.z;
                            v[j + 3] = __uint_as_float(r[j + 3]) + b.w;
                        }
                        if (kMode == kRowAdd) {
                            tma_store_wait_read<0>();
                            __syncwarp();
#pragma unroll
                            for (int j = 0; j < kParts; ++j) {
                                const int px = j * (32 / kParts) + lane / kParts;
                                const int psw = kG == 32 ? (px >> 1) & 3 : (px >> 2) & 1;
                                reinterpret_cast<uint4*>(sbuf)[px * kParts + ((lane % kParts) ^ psw)] = add[j];
                            }
                            __syncwarp();
#pragma unroll
                            for (int j = 0; j < kParts; ++j) {
                                const uint4 w4 = sb[j ^ sw];
                                const uint32_t w[4] = {w4.x, w4.y, w4.z, w4.w};
#pragma unroll
                                for (int k = 0; k < 4; ++k) {
                                    v[8 * j + 2 * k] += __uint_as_float(w[k] << 16);
                                    v[8 * j + 2 * k + 1] += __uint_as_float(w[k] & 0xFFFF0000u);
                                }
                            }
                        }
                        if (kMode == kRowF32) {
                            if (relu) {
#pragma unroll
                                for (int j = 0; j < kG; ++j) v[j] = fmaxf(v[j], 0.0f);
                            }
                            if (x < a.W && y < a.H) {
                                float* d = reinterpret_cast<float*>(a.out) +
                                           (((size_t)img * a.H + y) * a.W + x) * a.out_c + a.out_off + c0;
#pragma unroll
                                for (int h = 0; h < kG; h += 16) {
                                    float w[16];
#pragma unroll
                                    for (int j = 0; j < 16; ++j) w[j] = v[h + j];
                                    store_f32(d + h, w, min(16, a.n_store - c0 - h));
                                }
                            }
                            continue;
                        }
#pragma unroll
                        for (int j = 0; j < kG / 2; ++j) pk[u][j] = pack_bf16x2(v[2 * j], v[2 * j + 1]);
                        if (relu) {   // of the rounded values: the same (a NaN becomes 0 either way)
#pragma unroll
                            for (int j = 0; j < kG / 2; ++j) pk[u][j] = relu2(pk[u][j]);
                        }
                        tma_store_wait_read<0>();   // the leader's last store has read the buffer
                        __syncwarp();
#pragma unroll
                        for (int j = 0; j < kG / 8; ++j)
                            sb[j ^ sw] = make_uint4(pk[u][4 * j], pk[u][4 * j + 1], pk[u][4 * j + 2], pk[u][4 * j + 3]);
                        fence_async_smem();
                        __syncwarp();
                        if (leader && y < a.H && x0 < a.W) {
                            tma_store_4d(&mo, sbuf, c0, x0, y, img);
                            if (a.up_out)
                                for (int k = 0; k < 4; ++k)
                                    tma_store_5d(&mu, sbuf, c0, k & 1, x0, 2 * y + (k >> 1), img);
                            tma_store_commit();
                        }
                    }
                    if (kMode == kRowPool) {
                        const int h2 = a.H >> 1, w2 = a.W >> 1, y2 = (yb * kR + o0) >> 1;
                        pool_store<kG>(pk[0], pk[kUnit - 1], y2 < h2 && (x >> 1) < w2,
                                       reinterpret_cast<__nv_bfloat16*>(a.pool_out) +
                                           (((size_t)img * h2 + y2) * w2 + (x >> 1)) * a.pool_c + a.pool_off + c0);
                    }
                }
            }
            if (!ok) break;
            if (++set == p.sets) {
                set = 0;
                phase ^= 1u;
            }
        }
        if (leader) tma_store_wait_all();
    }
    __syncthreads();
    if (warp == 1) tmem_dealloc(tmem, 512u);
}

// ---------------------------------------------------------------------------------------------
// 16 x 16-pixel tiles with streamed weights, for the layers whose weights do not fit in shared memory beside
// a row tile's chunks (sums by horizontal tap). A stage holds 64 input channels at one horizontal shift: the box {64 channels,
// 16 x, 18 y} in 128-byte-swizzled rows, whose windows from image row 0, 1 and 2 are the vertical taps,
// and the three taps' weights {64, Cout}. Both halves of the tile (16 x 8 pixels, M = 128, an accumulator
// each, with an issuer of its own) use them: 12 MMAs an issuer and stage.
// What bounds it: the TMA unit, which takes about 1.6 cycles for a box row of 64 bytes and 1.8 for one of
// 128, and the operand reads. A 16 x 8 tile with stages of 32 channels loads 352 rows for 288 cycles of
// MMAs (64 output channels); here it is 480 rows for 1152. Before and after, cold: 160 -> 64 channels on 540 x
// 960 pixels 103 -> 88 us, 224 -> 96 on 270 x 480 54 -> 46, 128 -> 96 on 2 x 300 x 300 44 -> 33.
constexpr int kBigEdge = 16;
constexpr int kBigXBytes = kBigEdge * (kBigEdge + 2) * 128;
constexpr int kBigMaxStages = 4;
constexpr int kBigThreads = 96 + 2 * kEpiThreads;   // producer, issuer, epilogue, issuer

struct BigPlan {
    int nx, ny, items;   // tiles per image row and column, in all
    int stages, groups;  // of four epilogue warps (two: one for each half)
};

template <int kG, bool kPool>
__global__ void __launch_bounds__(kBigThreads, 1) k_conv_tiles(const __grid_constant__ CUtensorMap mx,
                                                               const __grid_constant__ CUtensorMap mw,
                                                               const __grid_constant__ CUtensorMap mo,
                                                               const __grid_constant__ CUtensorMap mu, ConvArgs a,
                                                               BigPlan p) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    const int kc = a.cin / 32, chunks = (kc + 1) / 2, nco = a.cout;
    const int b_bytes = nco * 128, stage_bytes = kBigXBytes + 3 * b_bytes;
    uint8_t* stores = smem + p.stages * stage_bytes;   // 64 kG bytes per epilogue warp
    float* bsm = reinterpret_cast<float*>(stores + p.groups * 4 * 64 * kG);
    uint64_t* full = reinterpret_cast<uint64_t*>(bsm + 128);
    uint64_t* empty = full + kBigMaxStages;
    uint64_t* sfull = empty + kBigMaxStages;   // a tile's sums are complete (two tiles alternate in TMEM)
    uint64_t* sempty = sfull + 2;              // and have been read
    uint64_t* fin = sempty + 2;
    uint32_t* tslot = reinterpret_cast<uint32_t*>(fin + 1);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tslot + 1);

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    if (tid == 0) {
        for (int s = 0; s < p.stages; ++s) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], 2);
        }
        for (int i = 0; i < 2; ++i) {
            mbar_init(&sfull[i], 2);
            mbar_init(&sempty[i], 8);   // four warps for each half
        }
        mbar_init(fin, 2);
        *abort_flag = 0;
        mbar_fence_init();
    }
    if (warp == 1) {
        tmem_alloc(tslot, 512u);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    grid_dep_launch();
    grid_dep_wait();
    // -0 adds nothing, not even to a -0
    for (int i = tid; i < nco; i += blockDim.x) bsm[i] = a.bias ? __ldg(a.bias + i) : -0.0f;
    __syncthreads();
    const uint32_t tmem = *tslot;
    const int per_img = p.nx * p.ny;

    if (warp == 0) {
        if (lane == 0) {   // producer
            int s = 0;
            uint32_t use = 0;
            bool ok = true;
            for (int t = blockIdx.x; t < p.items && ok; t += gridDim.x) {
                const int img = t / per_img, r = t - img * per_img, ty = r / p.nx;
                const int x = (r - ty * p.nx) * kBigEdge - 1, y = ty * kBigEdge - 1;
                for (int dx = 0; dx < 3 && ok; ++dx)
                    for (int c = 0; c < chunks; ++c) {
                        if (use > 0) ok = mbar_wait_bounded(&empty[s], (use - 1u) & 1u, a.err);
                        if (!ok || *abort_flag) {
                            *abort_flag = 1;
                            ok = false;
                            break;
                        }
                        uint8_t* sa = smem + s * stage_bytes;
                        mbar_expect_tx(&full[s], (uint32_t)stage_bytes);
                        tma_load_4d(sa, &mx, 64 * c, x + dx, y, img, &full[s]);
                        for (int dy = 0; dy < 3; ++dy)
                            tma_load_2d(sa + kBigXBytes + dy * b_bytes, &mw, (3 * dy + dx) * a.cin + 64 * c, 0, &full[s]);
                        if (++s == p.stages) {
                            s = 0;
                            ++use;
                        }
                    }
            }
            // no load may be in flight when the CTA ends, whoever gave up
            for (int i = 0; i < p.stages; ++i) {
                const uint32_t uses = use + (i < s ? 1u : 0u);
                if (uses > 0) mbar_wait_bounded(&full[i], (uses - 1u) & 1u, a.err);
            }
        }
    } else if (warp == 1 || warp == 2 + 4 * p.groups) {
        // one MMA issuer for each half of the tile: the warp walks the stages, one elected lane issues
        constexpr uint32_t kHi = (1024u >> 4) | (1u << 14) | (2u << 29);   // 8-row groups 1 KB apart, SWIZZLE_128B
        const bool leader = elect_one();
        const uint32_t idesc = umma_idesc_bf16(128u, (uint32_t)nco), bstep = (uint32_t)b_bytes >> 4;
        const uint32_t slo = (smem_u32(smem) >> 4) | (1u << 16);
        int s = 0, kt = 0;
        uint32_t use = 0;
        bool ok = true;
        const int half = warp == 1 ? 0 : 1;
        // the taps dy of one 32-channel half of a stage
        auto chunk = [&](uint32_t d, uint32_t al, uint32_t bl, bool fresh) {
#pragma unroll
            for (int dy = 0; dy < 3; ++dy)
#pragma unroll
                for (int kk = 0; kk < 2; ++kk)
                    umma_bf16_lo(d, al + (uint32_t)(dy * kBigEdge * 8 + 2 * kk), kHi,
                                 bl + (uint32_t)dy * bstep + 2u * (uint32_t)kk, kHi, idesc,
                                 dy == 0 && kk == 0 && fresh ? 0u : 1u);
        };
        for (int t = blockIdx.x; t < p.items && ok; t += gridDim.x, ++kt) {
            const int set = kt & 1;
            const uint32_t d = tmem + (uint32_t)((set * 2 + half) * nco);
            if (kt >= 2) ok = mbar_wait_bounded(&sempty[set], (uint32_t)((kt >> 1) - 1) & 1u, a.err);
            for (int i = 0, c = 0; i < 3 * chunks && ok; ++i) {
                ok = mbar_wait_bounded(&full[s], use & 1u, a.err) && ok;
                ok = __all_sync(0xFFFFFFFFu, ok);
                if (!ok) break;
                tc_fence_after();
                if (leader) {
                    const uint32_t st = slo + (uint32_t)(s * (stage_bytes >> 4)), bl = st + (uint32_t)(kBigXBytes >> 4);
                    const uint32_t al = st + (uint32_t)(8 * half * kBigEdge * 8);
                    chunk(d, al, bl, i == 0);
                    if (2 * c + 1 < kc) chunk(d, al + 4u, bl + 4u, false);
                    umma_commit(&empty[s]);
                }
                __syncwarp();
                if (++s == p.stages) {
                    s = 0;
                    ++use;
                }
                if (++c == chunks) c = 0;
            }
            if (!ok) break;
            if (leader) umma_commit(&sfull[set]);
            __syncwarp();
        }
        if (!ok) *abort_flag = 1;
        if (leader) {
            umma_commit(fin);
            mbar_wait_bounded(fin, 0u, a.err);   // nothing may be in flight when TMEM is freed
        }
        __syncwarp();
    } else {
        const int q = warp & 3, group = (warp - 2) >> 2;
        uint8_t* sbuf = stores + (warp - 2) * 64 * kG;
        const uint32_t lane0 = tmem + ((uint32_t)(q * 32) << 16);
        const bool relu = (a.flags & kConvRelu) != 0, leader = elect_one();
        constexpr int kParts = kG / 8;   // 16-byte parts of a pixel's group of columns
        const int sw = kG == 32 ? (lane >> 1) & 3 : (lane >> 2) & 1;
        uint4* sb = reinterpret_cast<uint4*>(sbuf) + lane * kParts;
        int kt = 0;
        bool ok = true;
        for (int t = blockIdx.x; t < p.items && ok; t += gridDim.x, ++kt) {
            const int set = kt & 1;
            const int img = t / per_img, r = t - img * per_img, ty = r / p.nx, x0 = (r - ty * p.nx) * kBigEdge;
            ok = mbar_wait_bounded(&sfull[set], (uint32_t)(kt >> 1) & 1u, a.err) && !*abort_flag;
            ok = __all_sync(0xFFFFFFFFu, ok);
            if (!ok) break;
            tc_fence_after();
            for (int half = group; half < 2; half += p.groups) {
                const int y0 = ty * kBigEdge + 8 * half + 2 * q;   // the warp's two rows of 16 pixels
#pragma unroll 1
                for (int c0 = 0; c0 < nco; c0 += kG) {
                    uint32_t v[kG];
                    const uint32_t col = lane0 + (uint32_t)((set * 2 + half) * nco + c0);
                    if constexpr (kG == 32) tmem_ld32(col, v);
                    else tmem_ld16(col, v);
                    tmem_ld_wait();
                    if (c0 + kG >= nco) {
                        tc_fence_before();
                        __syncwarp();
                        if (leader) mbar_arrive(&sempty[set]);
                    }
                    const float4* b4 = reinterpret_cast<const float4*>(bsm + c0);
                    uint32_t pk[kG / 2];
#pragma unroll
                    for (int j = 0; j < kG; j += 4) {
                        const float4 b = b4[j / 4];
                        pk[j / 2] = pack_bf16x2(__uint_as_float(v[j]) + b.x, __uint_as_float(v[j + 1]) + b.y);
                        pk[j / 2 + 1] = pack_bf16x2(__uint_as_float(v[j + 2]) + b.z, __uint_as_float(v[j + 3]) + b.w);
                    }
                    if (relu) {   // of the rounded values: the same (a NaN becomes 0 either way)
#pragma unroll
                        for (int j = 0; j < kG / 2; ++j) pk[j] = relu2(pk[j]);
                    }
                    tma_store_wait_read<0>();   // the leader's last store has read the buffer
                    __syncwarp();
#pragma unroll
                    for (int j = 0; j < kParts; ++j)
                        sb[j ^ sw] = make_uint4(pk[4 * j], pk[4 * j + 1], pk[4 * j + 2], pk[4 * j + 3]);
                    fence_async_smem();
                    __syncwarp();
                    if (leader && y0 < a.H) {
                        tma_store_4d(&mo, sbuf, c0, x0, y0, img);
                        if (a.up_out)
                            for (int k = 0; k < 8; ++k)
                                if (y0 + (k >> 2) < a.H)
                                    tma_store_5d(&mu, sbuf + (k >> 2) * 32 * kG, c0, k & 1, x0,
                                                 2 * (y0 + (k >> 2)) + ((k >> 1) & 1), img);
                        tma_store_commit();
                    }
                    if (kPool) {
                        // the warp's 8 pooled pixels from their four stored values: lane l takes part
                        // l % 4 of pixel l / 4 (8 channels of 32, 4 of 16)
                        const int pp = lane >> 2, x = (x0 >> 1) + pp;
                        float lo[kParts], hi[kParts];
#pragma unroll
                        for (int j = 0; j < kParts; ++j) lo[j] = hi[j] = 0.0f;
#pragma unroll
                        for (int k = 0; k < 4; ++k) {
                            const int n = 2 * pp + (k & 1) + 16 * (k >> 1);
                            const int nsw = kG == 32 ? (n >> 1) & 3 : (n >> 2) & 1;
                            const int part = kG == 32 ? lane & 3 : (lane & 3) >> 1;
                            const uint32_t* w = reinterpret_cast<const uint32_t*>(sbuf + n * 2 * kG + 16 * (part ^ nsw)) +
                                                (kG == 32 ? 0 : 2 * (lane & 1));
#pragma unroll
                            for (int j = 0; j < kParts; ++j) {
                                lo[j] = lo[j] + __uint_as_float(w[j] << 16);
                                hi[j] = hi[j] + __uint_as_float(w[j] & 0xFFFF0000u);
                            }
                        }
                        if ((y0 >> 1) < (a.H >> 1) && x < (a.W >> 1)) {
                            uint32_t o[kParts];
#pragma unroll
                            for (int j = 0; j < kParts; ++j) o[j] = pack_bf16x2(lo[j] * 0.25f, hi[j] * 0.25f);
                            __nv_bfloat16* d = reinterpret_cast<__nv_bfloat16*>(a.pool_out) +
                                               (((size_t)img * (a.H >> 1) + (y0 >> 1)) * (a.W >> 1) + x) * a.pool_c +
                                               a.pool_off + c0 + 2 * kParts * (lane & 3);
                            if constexpr (kG == 32) *reinterpret_cast<uint4*>(d) = make_uint4(o[0], o[1], o[2], o[3]);
                            else *reinterpret_cast<uint2*>(d) = make_uint2(o[0], o[1]);
                        }
                        __syncwarp();
                    }
                }
            }
        }
        if (leader) tma_store_wait_all();
    }
    __syncthreads();
    if (warp == 1) tmem_dealloc(tmem, 512u);
}

}  // namespace

}  // namespace gk

using namespace gk;

cudaError_t gkrt_encode_tmap_bf16(CUtensorMap* map, const void* base, uint32_t rank, const uint64_t* dims,
                                  const uint64_t* strides_bytes, const uint32_t* box);
cudaError_t gkrt_encode_tmap_bf16_sw32(CUtensorMap* map, const void* base, uint32_t rank, const uint64_t* dims,
                                       const uint64_t* strides_bytes, const uint32_t* box);
cudaError_t gkrt_encode_tmap_bf16_sw128(CUtensorMap* map, const void* base, uint32_t rank, const uint64_t* dims,
                                        const uint64_t* strides_bytes, const uint32_t* box);
cudaError_t gkrt_encode_tmap_bf16_dense(CUtensorMap* map, const void* base, uint32_t rank, const uint64_t* dims,
                                        const uint64_t* strides_bytes, const uint32_t* box);

// Halo tiles for outputs of up to 32 channels whose weights (9 Cin Cout bf16) fit in 96 KB.
// The 1080p forward (event-timed, one box): row-box stages everywhere 1.560 ms; halo tiles for
// Cout <= 32 1.503 ms; also for Cout <= 64 with weights <= 40 KB 1.504 ms, <= 96 KB 1.556 ms
// (the 64 -> 64 layers then run one CTA per SM behind 72 KB of weights).
static bool conv_halo(int cin, int cout) { return cout <= 32 && 9 * cin * cout * 2 <= kHaloWeightMax; }
static size_t conv_halo_smem(int cin, int cout) {
    return (size_t)9 * cin * cout * 2 + kHaloStages * kHaloStage + (2 * kHaloStages + 6) * 8 + 8 + kEpiBuf + 1024;
}

constexpr int kRowSmem = 227 * 1024;
constexpr int kRowSmemMin = 116 * 1024;   // more than half of an SM's: one CTA per SM (it takes all of TMEM)
// Rows of a tile: 2 where its chunks stay in shared memory together or are several, or rows are pooled in
// pairs, else 3: four boxes are to fit. (Per output row of 32 -> 32 channels, 2 rows take 528 cycles of
// operand reads, 3 464, 4 432, taps of its own MMAs 720.)
static int row_rows(const ConvArgs& a, bool dx_outer) { return dx_outer || a.pool_out || a.cin > 32 ? 2 : 3; }

static size_t row_smem(const ConvArgs& a, const RowPlan& p, int stage) {
    return (size_t)9 * a.cin * a.cout * 2 + (size_t)2 * p.ring * stage + (size_t)p.groups * 4 * 64 * (a.cout % 32 ? 16 : 32) +
           128 * 4 + (2 * kRowMaxStages + 2 * kRowMaxSets + 3 * kRowMaxChunks + 1) * 8 + 8 + 1024;
}

// A barrier tells its phases apart by parity, so an epilogue group has to have seen a set's last use, or
// a later tile of the same issuer, before it waits for the next: with `units` turns a tile, a group is
// back at the same place of a tile after groups / gcd(groups, 2 units) of an issuer's tiles, of which
// there are to be no more than the issuer has sets.
static bool row_turns_ok(const RowPlan& p, int units) {
    return p.groups / std::gcd(p.groups, 2 * units) <= p.sets / 2;
}

// The plan of a convolution on row tiles, or none (items 0) where it does not fit or the other kernels'
// 16 x 8 tiles are estimated faster. Each issuer needs room for all of a tile's chunks where they stay,
// else for two. (Splitting the output channels over CTAs to make room was slower than 16 x 16 tiles with
// streamed weights: 64 -> 96 channels on 4 x 200 x 500 pixels 52 us, and 41.)
// The estimate is in times of one 16 x 8 tile per SM, of which the other kernels take their tiles' number
// over the SMs; a row tile was measured at 1.0 of those (128 x 2 pixels, sums by horizontal tap), 1.8 (128
// x 3, sums by chunk) and 1.5 (128 x 2), and whole waves count. Over the layers on 50 sizes from 16 x 32 to
// 4 x 200 x 500 either side of that line differs by at most 15% (64 -> 64 channels: 200 x 128 pixels 8.2 us
// by tiles, 7.9 by rows; 4 x 200 x 140 14.8 and 16.4).
static RowPlan row_plan(const ConvArgs& a, int rb, int sms) {
    RowPlan p{};
    const int kc = a.cin / 32;
    const bool dx_outer = !conv_halo(a.cin, a.cout);
    const int R = row_rows(a, dx_outer), stage = row_stage_bytes(rb, R), need = dx_outer ? kc : 2;
    if (a.cout > 128 || kc > kRowMaxChunks || (a.add_par && (a.pool_out || dx_outer))) return p;
    p.nxs = (a.W + 127) / 128;
    p.nyb = (a.H + R - 1) / R;
    const long long items = (long long)a.B * p.nxs * p.nyb;
    if (items > 0x7FFFFFFFLL / 4) return p;
    p.sets = std::min(kRowMaxSets, 512 / (R * a.cout)) & ~1;   // the issuers' in turn
    for (p.groups = kRowGroups; p.groups > 0; p.groups /= 2) {
        const size_t fixed = row_smem(a, p, 0);
        p.ring = fixed < (size_t)kRowSmem
                     ? std::min(kRowMaxStages / 2, (int)(((size_t)kRowSmem - fixed) / (2 * (size_t)stage)))
                     : 0;
        if (p.ring >= need && row_turns_ok(p, R / (a.pool_out ? 2 : 1))) break;
    }
    if (!p.groups) return p;
    const long long waves = (items + sms - 1) / sms;
    const float rows = dx_outer ? (float)waves + 0.3f : (R == 3 ? 1.8f : 1.5f) * (float)waves + 1.6f;
    const long long tiles = (long long)a.B * ((a.W + kTileX - 1) / kTileX) * ((a.H + kTileY - 1) / kTileY);
    if (rows < (float)tiles / (float)sms) p.items = (int)items;
    return p;
}

// For the tests: the row tiles that a convolution takes on a device of `sms`, 0 where it takes others.
extern "C" int gkrt_internal_conv_row_tiles(int B, int H, int W, int cin, int cout, int pooled, int sms) {
    ConvArgs a{};
    a.B = B; a.H = H; a.W = W; a.cin = cin; a.cout = cout;
    a.pool_out = pooled ? &a : nullptr;
    return row_plan(a, 64, sms).items;
}

// The tensor maps of a bf16 output's stores, kg channels of bx x by pixels, and of its nearest
// upsampling's, bx pixels of a row to every other pixel.
static cudaError_t encode_outputs(const ConvArgs& a, int kg, uint32_t bx, uint32_t by, CUtensorMap* mo, CUtensorMap* mu) {
    auto encode = kg == 32 ? gkrt_encode_tmap_bf16 : gkrt_encode_tmap_bf16_sw32;
    const uint64_t W = (uint64_t)a.W, H = (uint64_t)a.H, B = (uint64_t)a.B, oc = (uint64_t)a.out_c * 2;
    const uint64_t od[4] = {(uint64_t)a.cout, W, H, B}, os[3] = {oc, W * oc, H * W * oc};
    const uint32_t ob[4] = {(uint32_t)kg, bx, by, 1};
    cudaError_t e = encode(mo, static_cast<uint8_t*>(a.out) + (size_t)a.out_off * 2, 4, od, os, ob);
    *mu = *mo;
    if (e != cudaSuccess || !a.up_out) return e;
    const uint64_t uc = (uint64_t)a.up_c * 2;
    const uint64_t ud[5] = {(uint64_t)a.cout, 2, W, 2 * H, B}, us[4] = {uc, 2 * uc, 2 * W * uc, 4 * H * W * uc};
    const uint32_t ub[5] = {(uint32_t)kg, 1, bx, 1, 1};
    return encode(mu, static_cast<uint8_t*>(a.up_out) + (size_t)a.up_off * 2, 5, ud, us, ub);
}

static cudaError_t launch_rows(const void* xbase, int xv, uint64_t xc, const void* w, const ConvArgs& a, const RowPlan& p,
                               int rb, int sms, int dev, cudaStream_t st) {
    const bool f32 = (a.flags & kConvF32Out) != 0, dx_outer = !conv_halo(a.cin, a.cout);
    const int kg = a.cout % 32 ? 16 : 32, R = row_rows(a, dx_outer);
    const uint64_t W = (uint64_t)a.W, H = (uint64_t)a.H, B = (uint64_t)a.B;
    CUtensorMap mx, mw, mo, mu;
    const uint64_t xd[4] = {(uint64_t)xv, W, H, B};
    const uint64_t xs[3] = {xc * 2, W * xc * 2, H * W * xc * 2};
    const uint32_t xb[4] = {(uint32_t)rb / 2, kRowPix, (uint32_t)R + 2, 1};
    cudaError_t e = rb == 64 ? gkrt_encode_tmap_bf16(&mx, xbase, 4, xd, xs, xb)
                             : gkrt_encode_tmap_bf16_sw32(&mx, xbase, 4, xd, xs, xb);
    if (e != cudaSuccess) return e;
    const uint64_t wd[2] = {(uint64_t)9 * a.cin, (uint64_t)a.cout};
    const uint64_t ws[1] = {(uint64_t)9 * a.cin * 2};
    const uint32_t wb[2] = {32, (uint32_t)a.cout};
    if ((e = gkrt_encode_tmap_bf16(&mw, w, 2, wd, ws, wb)) != cudaSuccess) return e;
    mo = mu = mw;
    if (!f32 && (e = encode_outputs(a, kg, 32, 1, &mo, &mu)) != cudaSuccess) return e;
    typedef void (*Kernel)(CUtensorMap, CUtensorMap, CUtensorMap, CUtensorMap, ConvArgs, RowPlan);
    // by pixel bytes, rows and order of the sums; column group; mode
#define GK_ROWS(rb, kg, r, dxo, add) \
    {k_conv_rows<rb, kg, r, dxo, kRowPlain>, r % 2 ? nullptr : k_conv_rows<rb, kg, 2, dxo, kRowPool>, \
     add ? k_conv_rows<rb, kg, r, false, kRowAdd> : nullptr, k_conv_rows<rb, kg, r, dxo, kRowF32>}
    static const Kernel kernels[5][2][4] = {{GK_ROWS(64, 16, 2, true, false), GK_ROWS(64, 32, 2, true, false)},
                                            {GK_ROWS(64, 16, 2, false, true), GK_ROWS(64, 32, 2, false, true)},
                                            {GK_ROWS(64, 16, 3, false, true), GK_ROWS(64, 32, 3, false, true)},
                                            {GK_ROWS(32, 16, 2, false, true), GK_ROWS(32, 32, 2, false, true)},
                                            {GK_ROWS(32, 16, 3, false, true), GK_ROWS(32, 32, 3, false, true)}};
#undef GK_ROWS
    const int mode = f32 ? kRowF32 : a.add_par ? kRowAdd : a.pool_out ? kRowPool : kRowPlain;
    const Kernel kernel = kernels[dx_outer ? 0 : R - 1 + (rb == 32 ? 2 : 0)][kg == 32][mode];
    static bool attr[kMaxDevices] = {};
    if (!attr[dev]) {
        for (int i = 0; i < 40; ++i)
            if ((&kernels[0][0][0])[i] &&
                (e = cudaFuncSetAttribute((const void*)(&kernels[0][0][0])[i], cudaFuncAttributeMaxDynamicSharedMemorySize,
                                          kRowSmem)) != cudaSuccess)
                return e;
        attr[dev] = true;
    }
    const size_t smem = row_smem(a, p, row_stage_bytes(rb, R));
    return launch_after(kernel, dim3((unsigned)std::min(p.items, sms)), 96 + p.groups * kEpiThreads, std::max(smem, (size_t)kRowSmemMin), st,
                        mx, mw, mo, mu, a, p);
}

static size_t big_smem(const ConvArgs& a, const BigPlan& p) {
    return (size_t)p.stages * (kBigXBytes + 3 * a.cout * 128) + (size_t)p.groups * 4 * 64 * (a.cout % 32 ? 16 : 32) +
           128 * 4 + (2 * kBigMaxStages + 5) * 8 + 8 + 1024;
}

// The 16 x 16-tile plan of a convolution whose sums are taken by horizontal tap, or none (items 0) where
// 16 x 8 tiles are estimated faster: a wave of these was measured at 1.4 to 1.65 times one of those per
// SM (seven layers, sizes from 16 x 32 to 4 x 200 x 500), which lose where the second wave is nearly
// empty (160 -> 64 channels on 200 x 192 pixels 12.4 us by 16 x 8 tiles, 14.7 by these; 500 wide 24.4 and
// 20.5) and never where there is one wave (9.3 and 11.0).
static BigPlan big_plan(const ConvArgs& a, int sms) {
    BigPlan p{};
    if (a.cout > 128 || conv_halo(a.cin, a.cout) || a.add_par || (a.flags & kConvF32Out)) return p;
    // two epilogue groups, unless one leaves room for a third stage
    for (p.stages = 4, p.groups = 2; big_smem(a, p) > (size_t)kRowSmem;) {
        if (p.groups == 2 && p.stages == 3) p.groups = 1;
        else {
            p.groups = 2;
            --p.stages;
        }
    }
    p.nx = (a.W + kBigEdge - 1) / kBigEdge;
    p.ny = (a.H + kBigEdge - 1) / kBigEdge;
    const long long items = (long long)a.B * p.nx * p.ny;
    if (items > 0x7FFFFFFFLL / 4) return p;
    const long long waves = (items + sms - 1) / sms;
    const long long tiles = (long long)a.B * ((a.W + kTileX - 1) / kTileX) * ((a.H + kTileY - 1) / kTileY);
    if (waves == 1 || 1.6f * (float)waves <= (float)tiles / (float)sms + 0.7f) p.items = (int)items;
    return p;
}

static cudaError_t launch_big(const void* xbase, int xv, uint64_t xc, const void* w, const ConvArgs& a, const BigPlan& p,
                              int sms, int dev, cudaStream_t st) {
    const int kg = a.cout % 32 ? 16 : 32;
    const uint64_t W = (uint64_t)a.W, H = (uint64_t)a.H, B = (uint64_t)a.B;
    CUtensorMap mx, mw, mo, mu;
    const uint64_t xd[4] = {(uint64_t)xv, W, H, B};
    const uint64_t xs[3] = {xc * 2, W * xc * 2, H * W * xc * 2};
    const uint32_t xb[4] = {64, kBigEdge, kBigEdge + 2, 1};
    cudaError_t e = gkrt_encode_tmap_bf16_sw128(&mx, xbase, 4, xd, xs, xb);
    if (e != cudaSuccess) return e;
    const uint64_t wd[2] = {(uint64_t)9 * a.cin, (uint64_t)a.cout};
    const uint64_t ws[1] = {(uint64_t)9 * a.cin * 2};
    const uint32_t wb[2] = {64, (uint32_t)a.cout};
    if ((e = gkrt_encode_tmap_bf16_sw128(&mw, w, 2, wd, ws, wb)) != cudaSuccess) return e;
    if ((e = encode_outputs(a, kg, 16, 2, &mo, &mu)) != cudaSuccess) return e;
    typedef void (*Kernel)(CUtensorMap, CUtensorMap, CUtensorMap, CUtensorMap, ConvArgs, BigPlan);
    static const Kernel kernels[2][2] = {{k_conv_tiles<16, false>, k_conv_tiles<16, true>},
                                         {k_conv_tiles<32, false>, k_conv_tiles<32, true>}};
    static bool attr[kMaxDevices] = {};
    if (!attr[dev]) {
        for (int i = 0; i < 4; ++i)
            if ((e = cudaFuncSetAttribute((const void*)kernels[i / 2][i % 2], cudaFuncAttributeMaxDynamicSharedMemorySize,
                                          kRowSmem)) != cudaSuccess)
                return e;
        attr[dev] = true;
    }
    const size_t smem = std::max(big_smem(a, p), (size_t)kRowSmemMin);
    return launch_after(kernels[kg == 32][a.pool_out != nullptr], dim3((unsigned)std::min(p.items, sms)),
                        96 + p.groups * kEpiThreads, smem, st, mx, mw, mo, mu, a, p);
}

// Outputs of up to 128 channels use the row-box stages (three vertical taps per box); the
// 1080p forward: none 1.94 ms, up to 64 channels 1.67 ms, up to 128 channels 1.58 ms.
static bool conv_rows(int cout) { return cout <= 128; }

// Four stages per CTA (three for row-box stages, which carry three taps each), so that several
// CTAs share an SM (as many as shared memory and the 512 TMEM columns allow): independent
// load/MMA/epilogue streams hide L2 latency better than deeper rings in fewer CTAs (measured
// on the level-0 layers: 1.74 -> 1.67 ms for the 1080p forward with three row-box stages).
static int conv_stages(int cout) { return conv_rows(cout) ? 3 : 4; }

size_t gkrt_conv_smem_bytes(int cout) {
    const bool rows = conv_rows(cout);
    const int stage = (kTileX * (rows ? kTileY + 2 : kTileY) * 64 + (rows ? 3 : 1) * cout * 64 + 1023) & ~1023;
    return (size_t)conv_stages(cout) * stage + 2 * conv_stages(cout) * 8 + 5 * 8 + 8 + kEpiBuf + 1024;
}

static size_t conv_smem_max() {
    size_t m = 0;
    for (int c = 16; c <= 256; c += 16) m = std::max(m, gkrt_conv_smem_bytes(c));
    return m;
}

cudaError_t gkrt_launch_conv3x3(const void* x, const void* w, const ConvArgs& args, cudaStream_t st) {
    const bool f32 = (args.flags & kConvF32Out) != 0;
    if (args.cin % 32 || args.cin < 32 || args.cout % 16 || args.cout < 16 || args.cout > 256 || args.B < 1 ||
        args.H < 1 || args.W < 1 || (!f32 && (args.out_c % 16 || args.out_off % 16)) ||
        args.out_off + (f32 ? args.n_store : args.cout) > args.out_c || (f32 && args.n_store > args.cout) ||
        ((uintptr_t)x & 15u) || ((uintptr_t)w & 15u) || ((uintptr_t)args.out & 15u) ||
        ((uintptr_t)args.bias & 15u) || args.x_off % 8 ||
        args.x_valid < 0 || args.x_valid > args.cin || (args.x_valid % 32 && args.x_valid != 16))
        return cudaErrorInvalidValue;
    const int xv = args.x_valid > 0 ? args.x_valid : args.cin;   // channels present; the rest are zeros
    // the 32-channel boxes end inside the map, except 16 channels of a 32-channel input (halo
    // tiles with 32-byte rows)
    const bool halo = conv_halo(args.cin, args.cout);
    if (xv % 32 && !(halo && args.cin == 32)) return cudaErrorInvalidValue;
    if (args.x_c > 0 && (args.x_c % 8 || args.x_off + xv > args.x_c)) return cudaErrorInvalidValue;
    if ((args.pool_out || args.up_out || args.add_par) && f32) return cudaErrorInvalidValue;
    if (args.add_par && ((args.H | args.W) & 1 || args.add_c % 8 || args.add_c < 4 * args.cout ||
                         ((uintptr_t)args.add_par & 15u)))
        return cudaErrorInvalidValue;
    if (args.pool_out && (args.pool_c % 8 || args.pool_off % 8 || args.pool_off + args.cout > args.pool_c ||
                          ((uintptr_t)args.pool_out & 15u)))
        return cudaErrorInvalidValue;
    if (args.up_out && (args.up_c % 8 || args.up_off % 8 || args.up_off + args.cout > args.up_c ||
                        ((uintptr_t)args.up_out & 15u)))
        return cudaErrorInvalidValue;
    CUtensorMap mx, mw;
    const uint64_t xc = (uint64_t)(args.x_c > 0 ? args.x_c : xv);
    // per device: SM count, the attributes set, resident CTAs per output width
    static int sms_dev[kMaxDevices] = {};
    static bool halo_attr[kMaxDevices] = {};
    static size_t smem_set[kMaxDevices] = {};
    static int per_sm_cache[kMaxDevices][257] = {};
    const int dev = current_device_slot();
    if (dev < 0) return cudaErrorInvalidDevice;
    if (!sms_dev[dev]) {
        const cudaError_t e0 = cudaDeviceGetAttribute(&sms_dev[dev], cudaDevAttrMultiProcessorCount, dev);
        if (e0 != cudaSuccess) return e0;
    }
    const int sms = sms_dev[dev];
    if (!(xv % 32) || xc == 16) {   // (a 16-channel input is the whole pixel)
        const int rb = xv == 16 ? 32 : 64;
        const RowPlan plan = row_plan(args, rb, sms);
        if (plan.items)
            return launch_rows(static_cast<const uint8_t*>(x) + (size_t)args.x_off * 2, xv, xc, w, args, plan, rb, sms,
                               dev, st);
    }
    if (halo) {
        // rows when a chunk is the whole pixel (64 bytes, or 32 for an input of 16 channels),
        // planes when the pixel is wider than the chunk
        const int rb = (int)xc * 2 == std::min(xv, 32) * 2 ? (xv == 16 ? 32 : 64) : 16;
        if (rb == 16 && xv % 32) return cudaErrorInvalidValue;
        const uint64_t xd[4] = {(uint64_t)xv, (uint64_t)args.W, (uint64_t)args.H, (uint64_t)args.B};
        const uint64_t xs[3] = {xc * 2, (uint64_t)args.W * xc * 2, (uint64_t)args.H * args.W * xc * 2};
        const uint32_t xb[4] = {(uint32_t)(rb == 16 ? 8 : rb / 2), kHaloBoxX, kHaloBoxY, 1};
        const void* xbase = static_cast<const uint8_t*>(x) + (size_t)args.x_off * 2;
        cudaError_t e = rb == 64   ? gkrt_encode_tmap_bf16(&mx, xbase, 4, xd, xs, xb)
                        : rb == 32 ? gkrt_encode_tmap_bf16_sw32(&mx, xbase, 4, xd, xs, xb)
                                   : gkrt_encode_tmap_bf16_dense(&mx, xbase, 4, xd, xs, xb);
        if (e != cudaSuccess) return e;
        const uint64_t wd[2] = {(uint64_t)9 * args.cin, (uint64_t)args.cout};
        const uint64_t ws[1] = {(uint64_t)9 * args.cin * 2};
        const uint32_t wb[2] = {32, (uint32_t)args.cout};
        if ((e = gkrt_encode_tmap_bf16(&mw, w, 2, wd, ws, wb)) != cudaSuccess) return e;
        const size_t smem = conv_halo_smem(args.cin, args.cout);
        if (!halo_attr[dev]) {
            const int mx_smem = (int)(kHaloWeightMax + kHaloStages * kHaloStage + 2048 + kEpiBuf);
            for (const void* f : {(const void*)k_conv3x3_halo<16>, (const void*)k_conv3x3_halo<32>,
                                  (const void*)k_conv3x3_halo<64>}) {
                if ((e = cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, mx_smem)) != cudaSuccess)
                    return e;
                if ((e = cudaFuncSetAttribute(f, cudaFuncAttributePreferredSharedMemoryCarveout,
                                              (int)cudaSharedmemCarveoutMaxShared)) != cudaSuccess)
                    return e;
            }
            halo_attr[dev] = true;
        }
        const int ncols = 2 * (args.cout <= 32 ? 32 : 64);
        const int per_sm = std::max(1, std::min({(int)((227 * 1024) / (smem + 1024)), 512 / ncols,
                                                 2048 / kConvThreads}));
        const int tiles_x = (args.W + kHaloX - 1) / kHaloX, tiles_y = (args.H + kHaloY - 1) / kHaloY;
        const int ntiles = tiles_x * tiles_y * args.B;
        const int grid = std::min(ntiles, sms * per_sm);
        const auto kernel = rb == 64 ? k_conv3x3_halo<64> : rb == 32 ? k_conv3x3_halo<32> : k_conv3x3_halo<16>;
        kernel<<<grid, kConvThreads, smem, st>>>(mx, mw, args, tiles_x, tiles_y, ntiles);
        return cudaGetLastError();
    }
    const uint64_t xd[4] = {(uint64_t)xv, (uint64_t)args.W, (uint64_t)args.H, (uint64_t)args.B};
    const uint64_t xs[3] = {xc * 2, (uint64_t)args.W * xc * 2, (uint64_t)args.H * args.W * xc * 2};
    const bool rows = conv_rows(args.cout);
    const uint32_t xb[4] = {32, kTileX, (uint32_t)(rows ? kTileY + 2 : kTileY), 1};
    const void* xbase = static_cast<const uint8_t*>(x) + (size_t)args.x_off * 2;
    cudaError_t e = gkrt_encode_tmap_bf16(&mx, xbase, 4, xd, xs, xb);
    if (e != cudaSuccess) return e;
    const uint64_t wd[2] = {(uint64_t)9 * args.cin, (uint64_t)args.cout};
    const uint64_t ws[1] = {(uint64_t)9 * args.cin * 2};
    const uint32_t wb[2] = {32, (uint32_t)args.cout};
    e = gkrt_encode_tmap_bf16(&mw, w, 2, wd, ws, wb);
    if (e != cudaSuccess) return e;
    const BigPlan big = big_plan(args, sms);
    if (big.items) return launch_big(xbase, xv, xc, w, args, big, sms, dev, st);
    const size_t smem = gkrt_conv_smem_bytes(args.cout);
    // launch geometry per output width, computed once per device (host calls kept off the
    // per-launch path)
    if (smem > smem_set[dev]) {
        for (const void* f : {(const void*)k_conv3x3<true>, (const void*)k_conv3x3<false>}) {
            if ((e = cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)conv_smem_max())) !=
                cudaSuccess)
                return e;
            if ((e = cudaFuncSetAttribute(f, cudaFuncAttributePreferredSharedMemoryCarveout,
                                          (int)cudaSharedmemCarveoutMaxShared)) != cudaSuccess)
                return e;
        }
        smem_set[dev] = conv_smem_max();
    }
    int per_sm = per_sm_cache[dev][args.cout];
    if (!per_sm) {
        // resident CTAs per SM: shared memory (227 KB per SM, 1 KB reserved per CTA), the 512
        // TMEM columns (two accumulators per CTA) and 2048 threads
        const int ncols = 2 * (args.cout <= 32 ? 32 : args.cout <= 64 ? 64 : args.cout <= 128 ? 128 : 256);
        per_sm = std::min({(int)((227 * 1024) / (smem + 1024)), 512 / ncols, 2048 / kConvThreads});
        per_sm = std::max(1, per_sm);
        per_sm_cache[dev][args.cout] = per_sm;
    }
    const int tiles_x = (args.W + kTileX - 1) / kTileX, tiles_y = (args.H + kTileY - 1) / kTileY;
    const int ntiles = tiles_x * tiles_y * args.B;
    const int grid = std::min(ntiles, sms * per_sm);
    const auto kernel = rows ? k_conv3x3<true> : k_conv3x3<false>;
    kernel<<<grid, kConvThreads, smem, st>>>(mx, mw, args, tiles_x, tiles_y, ntiles, conv_stages(args.cout));
    return cudaGetLastError();
}
