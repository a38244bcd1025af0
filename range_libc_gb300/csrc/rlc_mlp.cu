// Learned range surrogate: a per-map MLP that predicts where a ray meets a
// wall, trained on rays cast by the exact GPU ray marcher, with hand-written
// tcgen05 (TMEM-accumulating) BF16 GEMMs for the forward and backward passes
// and an Adam kernel.  No counterpart in the reference.
//
// Model: the grid-frame ray (x, y, theta) becomes u = (x/W, y/H, cos, sin);
// each of the 4 inputs is expanded by 64 sinusoidal frequencies f_k =
// fmax^(k/63) (sin and cos of pi f_k u) into 512 features, then four hidden
// layers of width 256 with GELU (tanh form), then one linear output: the
// march parameter t at which the exact marcher reaches its hit cell (pixels).
// Weights and activations are BF16, accumulation and the output layer FP32.
//
// A prediction t^ is accepted when the cell at x0 + t^ dir is occupied and
// the cell at x0 + (t^ - 1) dir is free; the range returned is then the
// reference's distance to that cell's corner, otherwise the ray is recast
// exactly (k_resolve, which collects a block's rejected rays and marches them).
#include "rangelibc.h"
#include "rlc_internal.cuh"
#include "rlc_tc.cuh"

#include <cuda.h>
#include <cuda_bf16.h>

#include <atomic>
#include <cmath>
#include <mutex>
#include <cstdio>
#include <cstring>
#include <vector>

#define TRY(x) do { cudaError_t _e = (x); if (_e != cudaSuccess) return _e; } while (0)

namespace rlc {
namespace {

typedef __nv_bfloat16 bf16;

constexpr int kFeat = 512;      // 4 inputs x 64 frequencies x {sin, cos}
constexpr int kHidden = 256;
constexpr int kLayers = 4;      // hidden layers
constexpr int kBM = 128;        // GEMM tile rows (TMEM lanes)
constexpr int kBN = 256;        // GEMM tile columns (TMEM columns)

// flat fp32 parameter layout
constexpr size_t kW0 = (size_t)kHidden * kFeat;              // layer 0: 256 x 512 (out x in)
constexpr size_t kWh = (size_t)kHidden * kHidden;            // layers 1-3: 256 x 256
constexpr size_t kParamCount = kW0 + kHidden + 3 * (kWh + kHidden) + kHidden + 1;

__host__ __device__ inline size_t w_offset(int l) { return l == 0 ? 0 : kW0 + kHidden + (size_t)(l - 1) * (kWh + kHidden); }
__host__ __device__ inline size_t b_offset(int l) { return w_offset(l) + (l == 0 ? kW0 : kWh); }
__host__ __device__ inline int layer_in(int l) { return l == 0 ? kFeat : kHidden; }
constexpr size_t kOutW = kW0 + kHidden + 3 * (kWh + kHidden);  // output weights [256], then bias [1]

// -------------------------------------------------------------------- GEMM
struct GemmArgs {
    const bf16* A;   // A[m * lda + k] (K-major), or with a_t A[k * lda + m] (M-major)
    const bf16* B;   // B[n * ldb + k], or with b_t B[k * ldb + n]
    int lda, ldb, a_t, b_t;
    int M, N, K;
    int ksplit;          // K range of blockIdx.z: [z * ksplit, min((z + 1) * ksplit, K))
    float* C;            // C[m * ldc + n], of split z at C + z * part_stride; 16-byte aligned
    int ldc;
    size_t part_stride;
    float* k_sums;       // with a_t: also the sums over k of A[k][m], at k_sums[z * part_stride + m]
    unsigned* err;
};

// GELU (tanh form).  tanh is the SFU's single-instruction approximation
// (PTX tanh.approx.f32, relative error about 2^-11, below the BF16 rounding
// of the activations); training and inference use the same function.
__device__ __forceinline__ float tanh_sfu(float x) {
    float y;
    asm("tanh.approx.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// Two floats per register pair: one issue slot for both (each rounded as by itself).  The network's
// elementwise work is issue-bound (k_top for 65,536 rays: 25.7 -> 23.8 us).
typedef unsigned long long f32x2;
__device__ __forceinline__ f32x2 pack2(float a, float b) {
    f32x2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ float2 unpack2(f32x2 v) {
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
    return r;
}
__device__ __forceinline__ f32x2 both(float a) { return pack2(a, a); }
__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b) {
    f32x2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b) {
    f32x2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
    f32x2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ f32x2 tanh2(f32x2 x) {
    const float2 v = unpack2(x);
    return pack2(tanh_sfu(v.x), tanh_sfu(v.y));
}
constexpr float kGelu0 = 0.7978845608028654f, kGelu1 = 0.044715f;

// The assembler contracts mul.rn.f32x2 + add.rn.f32x2 to one rounding, also without -fmad.  A product
// that is added to something is therefore an fma with a -0 that it cannot see: a * b rounded as by itself.
__constant__ float c_neg_zero = -0.0f;
__device__ __forceinline__ f32x2 mul2_then(f32x2 a, f32x2 b) { return fma2(a, b, both(c_neg_zero)); }

// tanh(k0 (z + k1 z^3))
__device__ __forceinline__ f32x2 gelu_tanh(f32x2 z) {
    return tanh2(mul2(both(kGelu0), add2(z, mul2_then(mul2(mul2(both(kGelu1), z), z), z))));
}
// 0.5 z (1 + tanh(..))
__device__ __forceinline__ float2 gelu(f32x2 z) {
    return unpack2(mul2(mul2(both(0.5f), z), add2(both(1.0f), gelu_tanh(z))));
}
// 0.5 (1 + th) + 0.5 z (1 - th^2) k0 (1 + 3 k1 z^2)
__device__ __forceinline__ f32x2 gelu_grad(f32x2 z) {
    const f32x2 one = both(1.0f), half = both(0.5f), th = gelu_tanh(z);
    const f32x2 sech2 = fma2(mul2(th, th), both(-1.0f), one);   // 1 - th * th, rounded as those two steps
    const f32x2 du = add2(one, mul2_then(mul2(both(3.0f * kGelu1), z), z));
    return add2(mul2_then(half, add2(one, th)), mul2_then(mul2(mul2(mul2(half, z), sech2), both(kGelu0)), du));
}

// --------------------------------------------------------------- TMA GEMM
// C tile [128 x BN] at (blockIdx.y * 128, blockIdx.x * BN) of C = A . B^T in fp32, K range
// [z * ksplit, min((z + 1) * ksplit, K)): the weight gradients, whose K is the batch.  Either operand
// may lie K-major or, as the batch's rows do here, M/N-major: the tensor cores read both, so no
// transposed copy of an activation or gradient is ever written (before, the epilogues stored a second
// copy two bytes at a time, and three transposes ran per step).
//
// Warp-specialised (10 warps, 192 KB of pipeline stages):
//   warp 0     TMA producer: per K chunk of KS, the tiles of A (128 rows or columns) and B (BN)
//              into stage s, completing on full[s]; it reuses a stage once the MMAs that read it have
//              committed to empty[s] (and the warps that sum it have arrived there);
//   warp 1     allocates BN TMEM columns; one thread issues the chunk's
//              tcgen05.mma (K = 16 each) per stage and commits them to empty[s], and after the
//              last chunk to `accum`;
//   warps 2-9  with k_sums: add up the rows of every stage of A on its way (the bias gradients, which
//              took four more passes over the gradients); then the epilogue: wait for `accum`, read
//              half of the columns of 32 rows of the accumulator with tcgen05.ld (warp w reads TMEM
//              lanes 32 (w % 4) .. + 31) and store it.
// Shared-memory operand layouts, 128-byte swizzle, as the TMA writes them: K-major, row r of a tile at
// r * 128 bytes (tc::make_desc_sw128); M/N-major, blocks of 64 columns, of which K row k lies at
// k * 128 bytes (tc::make_desc_sw128_mn); 16-byte chunks permuted by the row & 7.
// Every wait is bounded (about a second); a time-out sets bit 16 of *err, the remaining roles stop
// at their next wait, and the CTA still frees its TMEM.
//
// KS: K of a stage.  64, or 128 where both operands are M/N-major and few CTAs each have a long chain:
// there the issuing threads set the pace (a step of 32,640 rays: 0.93 ms in stages of 64, 0.84 in stages of
// 128, 0.78 with the issuing warps kept together, so that their loops run in uniform registers).
//
// Bound by reading dZ and the layer's input: 67 MB for a hidden layer and 65,536 rays, 17 us (22 from the
// transposed copies, which cost 32 us and more to write, and 27 us for the bias sums).
constexpr uint32_t kStageA = kBM * tc::kKChunk * 2;   // 16 KB
constexpr uint32_t kBlockMN = 64 * tc::kKChunk * 2;   // an M/N-major block of 64 columns x 64 K: 8 KB
constexpr size_t kGemmSmem = 196608 + 1024;           // the stages, + alignment slack
constexpr int kEpiWarps = 8;
constexpr int kGemmThreads = 64 + 32 * kEpiWarps;

// 32 bytes per lane and instruction: whole sectors although the lanes' rows lie apart
__device__ __forceinline__ void store32(void* p, const uint32_t* v) {
    asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(p), "r"(v[0]), "r"(v[1]), "r"(v[2]),
                 "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7])
                 : "memory");
}
__device__ __forceinline__ void load32(const void* p, uint32_t* v) {
    asm volatile("ld.global.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7])
                 : "l"(p));
}
__device__ __forceinline__ bool same_bits(float a, float b) { return __float_as_uint(a) == __float_as_uint(b); }
__device__ __forceinline__ uint32_t pack_bf16(float a, float b) {
    const __nv_bfloat162 v = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<const uint32_t*>(&v);
}
__device__ __forceinline__ f32x2 widen_bf16(uint32_t u) {
    f32x2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "r"(u << 16), "r"(u & 0xffff0000u));
    return r;
}
__device__ __forceinline__ float2 unpack_bf16(uint32_t u) { return __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&u)); }

template <int BN, int KS>
__global__ void __launch_bounds__(kGemmThreads, 1)
k_gemm_tma(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, GemmArgs g) {
    constexpr uint32_t kStageA = kBM * KS * 2, kStageB = BN * KS * 2, kBlock = 64 * KS * 2;   // kBlock: 64 columns, M/N-major
    constexpr int kStages = 196608 / (kStageA + kStageB);
    extern __shared__ uint8_t smem_raw[];
    __shared__ __align__(8) uint64_t full[kStages], empty[kStages], accum;
    __shared__ uint32_t tmem_base;
    __shared__ int abort_flag, n_issued, n_consumed;
    __shared__ __align__(16) float s_sums[kEpiWarps / 2][kBM];
    uint8_t* smem = reinterpret_cast<uint8_t*>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    const uint32_t sbase = tc::smem_addr(smem);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int m0 = blockIdx.y * kBM, n0 = blockIdx.x * BN;
    const int kbase = blockIdx.z * g.ksplit;
    const int nchunks = min(g.ksplit, g.K - kbase) / KS;
    const bool sums = g.k_sums != nullptr && g.a_t && blockIdx.x == 0;
    if (warp == 1) tc::tmem_alloc(tc::smem_addr(&tmem_base), BN);
    if (threadIdx.x == 0) {
        for (int i = 0; i < kStages; ++i) {
            tc::mbar_init(tc::smem_addr(&full[i]), 1);
            tc::mbar_init(tc::smem_addr(&empty[i]), sums ? 1 + kEpiWarps : 1);   // the MMAs' commit, and the summing warps
        }
        tc::mbar_init(tc::smem_addr(&accum), 1);
        abort_flag = 0;
        n_issued = 0;
        n_consumed = 0;
        tc::fence_mbar_init();
    }
    after_previous();
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    const uint32_t tmem = tmem_base;
    auto stage_a = [&](int st) { return sbase + (uint32_t)st * (kStageA + kStageB); };
    auto stage_b = [&](int st) { return stage_a(st) + kStageA; };
    if (warp == 0) {
        // ---- producer; the warp keeps together, so that the loop runs in uniform registers
        tc::tma_prefetch_map(&tmA);
        tc::tma_prefetch_map(&tmB);
        int c = 0;
        for (int st = 0, phase = 1, k = kbase; c < nchunks; ++c, k += KS) {
            if (c >= kStages && !__all_sync(0xffffffffu, tc::mbar_wait(tc::smem_addr(&empty[st]), phase))) {
                if (lane == 0) {
                    atomicOr(g.err, 16u);
                    atomicExch(&abort_flag, 1);
                }
                break;
            }
            const uint32_t fb = tc::smem_addr(&full[st]);
            if (tc::elect_one()) {
                tc::mbar_arrive_expect_tx(fb, kStageA + kStageB);
                tc::tma_load_3d(stage_a(st), &tmA, g.a_t ? 0 : k, g.a_t ? k : m0, g.a_t ? m0 / 64 : 0, fb);
                tc::tma_load_3d(stage_b(st), &tmB, g.b_t ? 0 : k, g.b_t ? k : n0, g.b_t ? n0 / 64 : 0, fb);
            }
            __syncwarp();
            if (++st == kStages) {
                st = 0;
                phase ^= 1;
            }
        }
        if (lane == 0) n_issued = c;
    } else if (warp == 1) {
        // ---- MMA issuer
        const uint32_t idesc = tc::make_idesc(kBM, BN) | (g.a_t ? tc::kIdescTransposeA : 0u) | (g.b_t ? tc::kIdescTransposeB : 0u);
        // descriptors of stage 0; a stage and a K step of 16 further are additions to their address field
        const uint64_t a0 = g.a_t ? tc::make_desc_sw128_mn(stage_a(0), kBlock) : tc::make_desc_sw128(stage_a(0));
        const uint64_t b0 = g.b_t ? tc::make_desc_sw128_mn(stage_b(0), kBlock) : tc::make_desc_sw128(stage_b(0));
        const uint32_t a_step = (g.a_t ? 16 * 128 : 32) >> 4, b_step = (g.b_t ? 16 * 128 : 32) >> 4;
        int c = 0;
        for (int st = 0, phase = 0; c < nchunks; ++c) {
            if (!__all_sync(0xffffffffu, tc::mbar_wait(tc::smem_addr(&full[st]), phase))) {
                if (lane == 0) {
                    atomicOr(g.err, 16u);
                    atomicExch(&abort_flag, 1);
                }
                break;
            }
            tc::fence_after_sync();
            const uint32_t at = (uint32_t)st * ((kStageA + kStageB) >> 4);
            if (tc::elect_one()) {
#pragma unroll
                for (int ks = 0; ks < KS / 16; ++ks)
                    tc::mma_bf16(tmem, a0 + (at + ks * a_step), b0 + (at + ks * b_step), idesc, (c > 0 || ks > 0) ? 1u : 0u);
                tc::mma_commit(tc::smem_addr(&empty[st]));
            }
            __syncwarp();
            if (++st == kStages) {
                st = 0;
                phase ^= 1;
            }
        }
        if (lane == 0) n_consumed = c;
        // `accum` completes once every MMA issued above has (also with none issued)
        if (tc::elect_one()) tc::mma_commit(tc::smem_addr(&accum));   // (the thread that issued them)
    } else if (warp >= 2) {
        if (sums) {
            // ---- sums over K of A's columns: two columns and a quarter of a stage's rows per thread
            constexpr int kRows = KS / (kEpiWarps / 2);
            const int pair = (threadIdx.x - 64) & 63, part = (threadIdx.x - 64) >> 6, r0 = part * kRows;
            const uint32_t at = (uint32_t)(pair >> 5) * kBlock + (uint32_t)(pair & 3) * 4u, chunk = (pair & 31) >> 2;
            float a0 = 0.0f, a1 = 0.0f;
            bool ok = true;
            for (int c = 0; c < nchunks && ok; ++c) {
                const int st = c % kStages;
                ok = __all_sync(0xffffffffu, tc::mbar_wait(tc::smem_addr(&full[st]), (c / kStages) & 1));
                if (ok) {
                    const uint8_t* tile = smem + (size_t)st * (kStageA + kStageB) + at;
#pragma unroll
                    for (int r = r0; r < r0 + kRows; ++r) {
                        const float2 v = unpack_bf16(*reinterpret_cast<const uint32_t*>(tile + r * 128 + ((chunk ^ (r & 7)) << 4)));
                        a0 += v.x;
                        a1 += v.y;
                    }
                }
                __syncwarp();
                if (lane == 0) tc::mbar_arrive(tc::smem_addr(&empty[st]));
            }
            if (!ok) {
                atomicOr(g.err, 16u);
                atomicExch(&abort_flag, 1);
            }
            // the parts of the rows, in a fixed order
            *reinterpret_cast<float2*>(&s_sums[part][2 * pair]) = make_float2(a0, a1);
            asm volatile("bar.sync 1, %0;" ::"n"(32 * kEpiWarps) : "memory");
            const int col = threadIdx.x - 64;
            if (col < kBM) {
                float sum = s_sums[0][col];
#pragma unroll
                for (int q = 1; q < kEpiWarps / 2; ++q) sum += s_sums[q][col];
                g.k_sums[(size_t)blockIdx.z * g.part_stride + m0 + col] = sum;
            }
        }
        // ---- epilogue
        const bool ok = __all_sync(0xffffffffu, tc::mbar_wait(tc::smem_addr(&accum), 0));
        tc::fence_after_sync();
        if (!ok) {
            if (lane == 0) atomicOr(g.err, 16u);
        } else if (!*(volatile int*)&abort_flag && nchunks > 0) {
            const int lq = warp & 3;   // TMEM lane quarter this warp may read
            const int row = m0 + lq * 32 + lane;
            const uint32_t lane_addr = tmem + ((uint32_t)(lq * 32) << 16);
            constexpr int kCols = BN / (kEpiWarps / 4);
            const int c0 = (warp - 2) / 4 * kCols;   // this warp's columns
            float* out = g.C + (size_t)blockIdx.z * g.part_stride + (size_t)row * g.ldc + n0;
            for (int cb = c0; cb < c0 + kCols; cb += 32) {
                float v[32];
                tc::tmem_ld32(lane_addr + cb, v);
                if (g.part_stride) {   // the workspace of partial sums
#pragma unroll
                    for (int i = 0; i < 32; i += 8) store32(out + cb + i, reinterpret_cast<const uint32_t*>(v + i));
                } else {
#pragma unroll
                    for (int i = 0; i < 32; i += 4)
                        *reinterpret_cast<float4*>(out + cb + i) = make_float4(v[i], v[i + 1], v[i + 2], v[i + 3]);
                }
            }
        }
    }
    tc::fence_before_sync();
    __syncthreads();
    if (abort_flag && threadIdx.x == 0) {
        // tile loads issued but never waited for are still landing in this CTA's shared memory:
        // wait for them (bounded) before the CTA exits
        for (int c = n_consumed; c < n_issued; ++c) (void)tc::mbar_wait(tc::smem_addr(&full[c % kStages]), (c / kStages) & 1);
    }
    __syncthreads();
    if (warp == 1) tc::tmem_dealloc(tmem, BN);
}

// cuTensorMapEncodeTiled through the runtime's driver entry point (no link to the driver library)
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn encode_tiled() {
    static EncodeTiledFn fn = nullptr;
    static std::once_flag once;
    std::call_once(once, [] {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q{};
        if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q) ==
                cudaSuccess && q == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<EncodeTiledFn>(p);
        else
            cudaGetLastError();
    });
    return fn;
}

// Tensor map of a bf16 operand of `rows` rows (or columns) x K with row stride ld, 128-byte swizzled in
// shared memory, as three dimensions so that one load brings a tile's K chunk either way: K-major
// {K, rows, 1} in boxes of 64 x box_rows; M/N-major (element (k, r) at k * ld + r) {64, K, rows / 64} in
// boxes of 64 x mn_k x box_rows / 64, blocks of 64 columns one after the other.  K-major only: the third
// dimension may count `batch` such operands, `pitch` elements apart.
cudaError_t operand_map(CUtensorMap* map, const bf16* base, bool mn_major, int rows, int K, int ld, int box_rows,
                        int batch = 1, size_t pitch = 64, int mn_k = tc::kKChunk) {
    EncodeTiledFn enc = encode_tiled();
    if (!enc) return cudaErrorNotSupported;
    if (((uintptr_t)base & 15) || (ld * 2) % 16 || (pitch * 2) % 16) return cudaErrorInvalidValue;
    const cuuint64_t dim[3] = {(cuuint64_t)(mn_major ? 64 : K), (cuuint64_t)(mn_major ? K : rows),
                               (cuuint64_t)(mn_major ? rows / 64 : batch)};
    const cuuint64_t stride[2] = {(cuuint64_t)ld * 2, (cuuint64_t)pitch * 2};
    const cuuint32_t box[3] = {64u, (cuuint32_t)(mn_major ? mn_k : box_rows), (cuuint32_t)(mn_major ? box_rows / 64 : 1)};
    const cuuint32_t estr[3] = {1, 1, 1};
    const CUresult r = enc(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<bf16*>(base), dim, stride, box, estr,
                           CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                           CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? cudaSuccess : cudaErrorInvalidValue;
}

template <int BN, int KS>
cudaError_t launch_gemm(const GemmArgs& g, cudaStream_t s) {
    CUtensorMap ta, tb;
    TRY(operand_map(&ta, g.A, g.a_t, g.M, g.K, g.lda, kBM, 1, 64, KS));
    TRY(operand_map(&tb, g.B, g.b_t, g.N, g.K, g.ldb, BN, 1, 64, KS));
    static std::atomic<unsigned long long> attr{0};
    TRY(ensure_smem_attr(k_gemm_tma<BN, KS>, (int)kGemmSmem, attr));
    return launch_next(k_gemm_tma<BN, KS>, dim3(g.N / BN, g.M / kBM, (g.K + g.ksplit - 1) / g.ksplit), kGemmThreads, kGemmSmem, s,
                       ta, tb, g);
}

// The widest tiles that still give two thirds of the SMs a CTA: A is read once per tile column, but a
// batch that splits badly (the single chain of an odd number of 128-ray tiles) leaves most SMs idle:
// two steps of 32,640 rays take 1.56 ms so (2.7 in 256-wide tiles, 2.5 before).
cudaError_t gemm(GemmArgs g, cudaStream_t s) {
    if (g.M % kBM || g.N % kBN || g.K % tc::kKChunk || g.K <= 0) return cudaErrorInvalidValue;
    if (g.ksplit <= 0) g.ksplit = g.K;
    if (g.ksplit % tc::kKChunk || (g.ksplit < g.K && !g.part_stride)) return cudaErrorInvalidValue;
    const long long tiles = (long long)(g.M / kBM) * (g.N / kBN) * ((g.K + g.ksplit - 1) / g.ksplit);
    if (tiles >= 96) return launch_gemm<256, 64>(g, s);
    if (tiles >= 48) return launch_gemm<128, 64>(g, s);
    return g.a_t && g.b_t && g.ksplit % 128 == 0 && g.K % 128 == 0 ? launch_gemm<64, 128>(g, s) : launch_gemm<64, 64>(g, s);
}

// ------------------------------------------------------------ layer GEMM
// The forward and input-gradient GEMMs of one layer: `rows` rows of A [rows x K] against the layer's
// weights, K = 512 or 256, as a persistent kernel, one CTA per SM.  Its weights (128 KB: all 256
// columns for K = 256, half of them for K = 512) stay in shared memory; the rows come through a ring
// of five 16 KB stages, and the accumulator has two buffers in TMEM, so that the tensor cores and the
// loads of the next 128 rows run beside the epilogue of these.  Bound by its bytes (a forward layer of
// 65,536 rays reads 33 and writes 67 MB); one CTA per tile, with its weights read again each time and
// nothing beside its epilogue, took 32 us for it (45-49 with the transposed copies), this 25; input gradients 46 -> 26.
//   FWD:  z = acc + bias, rounded to bf16, to Zout; GELU of it to Hout.  Weights [out x in], K-major.
//   else: acc * GELU'(Zin) to dZ.  The weights as they lie, [K = out][N = in]: N-major.
// Roles as in k_gemm_tma; the waits are bounded in the same way.
struct LayerArgs {
    int rows;
    const float* bias;   // FWD
    bf16 *Zout, *Hout;
    const bf16* Zin;     // input gradients
    bf16* dZ;
    unsigned* err;
};
constexpr int kLayerStages = 5;
constexpr uint32_t kWeightBytes = 131072;
constexpr size_t kLayerSmem = kWeightBytes + kLayerStages * (size_t)kStageA + 1024;

template <int BN, int K, bool FWD>
__global__ void __launch_bounds__(kGemmThreads, 1)
k_layer(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmW, LayerArgs g) {
    static_assert(BN * K * 2 == kWeightBytes && kHidden % BN == 0, "weights of a CTA");
    constexpr int kChunks = K / tc::kKChunk, kParts = kHidden / BN;
    constexpr uint32_t kWChunk = BN * tc::kKChunk * 2;
    extern __shared__ uint8_t smem_raw[];
    __shared__ __align__(8) uint64_t full[kLayerStages], empty[kLayerStages], wfull[kChunks], acc_full[2], acc_empty[2], drained;
    __shared__ uint32_t tmem_base;
    __shared__ int abort_flag, n_issued, n_consumed;
    __shared__ __align__(16) float s_bias[BN];
    uint8_t* smem = reinterpret_cast<uint8_t*>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    const uint32_t sW = tc::smem_addr(smem), sA = sW + kWeightBytes;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int n0 = (int)(blockIdx.x % kParts) * BN;
    const int tile0 = blockIdx.x / kParts, tiles = g.rows / kBM, step = gridDim.x / kParts;
    if (warp == 1) tc::tmem_alloc(tc::smem_addr(&tmem_base), 2 * BN);
    if (threadIdx.x == 0) {
        for (int i = 0; i < kLayerStages; ++i) {
            tc::mbar_init(tc::smem_addr(&full[i]), 1);
            tc::mbar_init(tc::smem_addr(&empty[i]), 1);
        }
        for (int c = 0; c < kChunks; ++c) tc::mbar_init(tc::smem_addr(&wfull[c]), 1);
        for (int i = 0; i < 2; ++i) {
            tc::mbar_init(tc::smem_addr(&acc_full[i]), 1);
            tc::mbar_init(tc::smem_addr(&acc_empty[i]), kEpiWarps);
        }
        tc::mbar_init(tc::smem_addr(&drained), 1);
        abort_flag = 0;
        n_issued = 0;
        n_consumed = 0;
        tc::fence_mbar_init();
    }
    after_previous();
    if (FWD)
        for (int i = threadIdx.x; i < BN; i += kGemmThreads) s_bias[i] = __ldg(g.bias + n0 + i);
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    const uint32_t tmem = tmem_base;
    auto aborted = [&]() { return *(volatile int*)&abort_flag != 0; };
    auto give_up = [&]() {
        atomicOr(g.err, 16u);
        atomicExch(&abort_flag, 1);
    };
    if (warp == 0 && lane == 0) {
        // ---- producer: the chunks of the CTA's row tiles, one after the other, go round the stages
        tc::tma_prefetch_map(&tmA);
        tc::tma_prefetch_map(&tmW);
        int n = 0, st = 0, phase = 1;
        bool ok = true;
        for (int t = tile0; t < tiles && ok; t += step) {
            for (int c = 0; c < kChunks; ++c, ++n) {
                if (n >= kLayerStages && !tc::mbar_wait(tc::smem_addr(&empty[st]), phase)) {
                    give_up();
                    ok = false;
                    break;
                }
                if (t == tile0) {   // the weights of this K chunk come with the first tile's
                    const uint32_t wb = tc::smem_addr(&wfull[c]);
                    tc::mbar_arrive_expect_tx(wb, kWChunk);
                    tc::tma_load_3d(sW + c * kWChunk, &tmW, FWD ? c * tc::kKChunk : 0, FWD ? n0 : c * tc::kKChunk, FWD ? 0 : n0 / 64, wb);
                }
                const uint32_t fb = tc::smem_addr(&full[st]);
                tc::mbar_arrive_expect_tx(fb, kStageA);
                tc::tma_load_3d(sA + st * kStageA, &tmA, c * tc::kKChunk, t * kBM, 0, fb);
                if (++st == kLayerStages) {
                    st = 0;
                    phase ^= 1;
                }
            }
        }
        n_issued = n;
    } else if (warp == 1 && lane == 0) {
        // ---- MMA issuer: the CTA's i-th tile accumulates in TMEM buffer i & 1
        const uint32_t idesc = tc::make_idesc(kBM, BN) | (FWD ? 0u : tc::kIdescTransposeB);
        const uint64_t a0 = tc::make_desc_sw128(sA);
        const uint64_t w0 = FWD ? tc::make_desc_sw128(sW) : tc::make_desc_sw128_mn(sW, kBlockMN);
        constexpr uint32_t kWStep = (FWD ? 32 : 16 * 128) >> 4;
        int n = 0, i = 0, st = 0, phase = 0;
        bool ok = true;
        for (int t = tile0; t < tiles && ok; t += step, ++i) {
            const uint32_t acc = tmem + (uint32_t)(i & 1) * BN;
            if (i >= 2) ok = tc::mbar_wait(tc::smem_addr(&acc_empty[i & 1]), ((i >> 1) - 1) & 1);
            tc::fence_after_sync();
            for (int c = 0; c < kChunks && ok; ++c) {
                if (i == 0) ok = tc::mbar_wait(tc::smem_addr(&wfull[c]), 0);
                if (ok) ok = tc::mbar_wait(tc::smem_addr(&full[st]), phase);
                if (!ok) break;
                tc::fence_after_sync();
#pragma unroll
                for (int ks = 0; ks < tc::kKChunk / 16; ++ks)
                    tc::mma_bf16(acc, a0 + (uint32_t)(st * (kStageA >> 4) + ks * 2), w0 + (c * (kWChunk >> 4) + ks * kWStep), idesc,
                                 (c > 0 || ks > 0) ? 1u : 0u);
                tc::mma_commit(tc::smem_addr(&empty[st]));
                ++n;
                if (++st == kLayerStages) {
                    st = 0;
                    phase ^= 1;
                }
            }
            if (ok) tc::mma_commit(tc::smem_addr(&acc_full[i & 1]));
        }
        n_consumed = n;
        if (!ok) {   // let what was issued end before the TMEM is freed
            give_up();
            tc::mma_commit(tc::smem_addr(&drained));
            (void)tc::mbar_wait(tc::smem_addr(&drained), 0);
        }
    } else if (warp >= 2) {
        // ---- epilogue
        constexpr int kCols = BN / (kEpiWarps / 4);
        const int lq = warp & 3, c0 = (warp - 2) / 4 * kCols;   // TMEM lane quarter and columns of this warp
        int i = 0;
        for (int t = tile0; t < tiles; t += step, ++i) {
            const size_t at = (size_t)(t * kBM + lq * 32 + lane) * kHidden + n0 + c0;
            uint32_t zin[16];
            if (!FWD) {
                load32(g.Zin + at, zin);
                load32(g.Zin + at + 16, zin + 8);
            }
            const bool ok = __all_sync(0xffffffffu, tc::mbar_wait(tc::smem_addr(&acc_full[i & 1]), (i >> 1) & 1) && !aborted());
            tc::fence_after_sync();
            if (!ok) {
                if (lane == 0) give_up();
                break;
            }
            const uint32_t acc = tmem + (uint32_t)(i & 1) * BN + ((uint32_t)(lq * 32) << 16) + c0;
#pragma unroll
            for (int cb = 0; cb < kCols; cb += 32) {
                float v[32];
                tc::tmem_ld32(acc + cb, v);
                if (cb + 32 == kCols) {   // the accumulator is read: the next but one tile may have it
                    tc::fence_before_sync();
                    __syncwarp();
                    if (lane == 0) tc::mbar_arrive(tc::smem_addr(&acc_empty[i & 1]));
                }
                if (FWD) {
                    uint32_t zp[16], hp[16];
#pragma unroll
                    for (int q = 0; q < 32; q += 4) {
                        const float4 b = *reinterpret_cast<const float4*>(s_bias + c0 + cb + q);
                        const float2 a0 = unpack2(add2(pack2(v[q], v[q + 1]), pack2(b.x, b.y)));
                        const float2 a1 = unpack2(add2(pack2(v[q + 2], v[q + 3]), pack2(b.z, b.w)));
                        zp[q / 2] = pack_bf16(a0.x, a0.y);
                        zp[q / 2 + 1] = pack_bf16(a1.x, a1.y);
                        // GELU of the stored (rounded) pre-activation
                        const float2 h0 = gelu(widen_bf16(zp[q / 2])), h1 = gelu(widen_bf16(zp[q / 2 + 1]));
                        hp[q / 2] = pack_bf16(h0.x, h0.y);
                        hp[q / 2 + 1] = pack_bf16(h1.x, h1.y);
                    }
                    store32(g.Zout + at + cb, zp);
                    store32(g.Zout + at + cb + 16, zp + 8);
                    store32(g.Hout + at + cb, hp);
                    store32(g.Hout + at + cb + 16, hp + 8);
                } else {
                    uint32_t dp[16];
#pragma unroll
                    for (int q = 0; q < 32; q += 2) {
                        const float2 d = unpack2(mul2(pack2(v[q], v[q + 1]), gelu_grad(widen_bf16(zin[q / 2]))));
                        dp[q / 2] = pack_bf16(d.x, d.y);
                    }
                    if (cb + 32 < kCols) {   // the next columns' pre-activations beside this store and TMEM read
                        load32(g.Zin + at + cb + 32, zin);
                        load32(g.Zin + at + cb + 48, zin + 8);
                    }
                    store32(g.dZ + at + cb, dp);
                    store32(g.dZ + at + cb + 16, dp + 8);
                }
            }
        }
    }
    tc::fence_before_sync();
    __syncthreads();
    if (abort_flag && threadIdx.x == 0) {
        // loads issued but never waited for are still landing in this CTA's shared memory: wait for
        // them (bounded) before the CTA exits
        for (int c = 0; c < min(kChunks, n_issued); ++c) (void)tc::mbar_wait(tc::smem_addr(&wfull[c]), 0);
        for (int n = n_consumed; n < n_issued; ++n)
            (void)tc::mbar_wait(tc::smem_addr(&full[n % kLayerStages]), (n / kLayerStages) & 1);
    }
    __syncthreads();
    if (warp == 1) tc::tmem_dealloc(tmem, 2 * BN);
}

// rows: a multiple of 128; A [rows x K], W the layer's weights [256 x K] (FWD) or [K][256]
template <int BN, int K, bool FWD>
cudaError_t layer(const bf16* A, const bf16* W, const LayerArgs& g, cudaStream_t s) {
    CUtensorMap ta, tw;
    TRY(operand_map(&ta, A, false, g.rows, K, K, kBM));
    TRY(operand_map(&tw, W, !FWD, kHidden, K, FWD ? K : kHidden, BN));
    static std::atomic<unsigned long long> attr{0};
    TRY(ensure_smem_attr(k_layer<BN, K, FWD>, (int)kLayerSmem, attr));
    constexpr int kParts = kHidden / BN;
    const int grid = std::min(152 / kParts, g.rows / kBM) * kParts;
    return launch_next(k_layer<BN, K, FWD>, dim3(grid), kGemmThreads, kLayerSmem, s, ta, tw, g);
}

// ---------------------------------------------------------------- features
struct FeatParams {
    float inv_w, inv_h;
    float freq[64];
};

// Features of grid-frame rays (x, y, theta), one row per warp at a time: lane l computes frequencies l
// and l + 32 of each input, so that a row's 1 KB leaves in whole lines (one row per thread before: 108
// us for 65,536 rows, now 22).  Rows from n on are zero.
constexpr int kFeatRows = 8;   // rows per warp

__global__ void __launch_bounds__(256) k_features(FeatParams fp, const float* xyt, int n, int n_pad,
                                                  bf16* __restrict__ X) {
    __shared__ float s_freq[64];
    if (threadIdx.x < 64) s_freq[threadIdx.x] = fp.freq[threadIdx.x];
    __syncthreads();
    const int lane = threadIdx.x & 31;
    const float f0 = s_freq[lane], f1 = s_freq[lane + 32];
    const int r0 = (blockIdx.x * 8 + (threadIdx.x >> 5)) * kFeatRows;
    after_previous();
    for (int r = r0; r < min(r0 + kFeatRows, n_pad); ++r) {
        uint32_t* out = reinterpret_cast<uint32_t*>(X + (size_t)r * kFeat) + lane;
        if (r >= n) {
#pragma unroll
            for (int j = 0; j < kFeat / 64; ++j) out[j * 32] = 0u;
            continue;
        }
        float s, c;
        sincosf(xyt[3 * (size_t)r + 2], &s, &c);
        const float u[4] = {xyt[3 * (size_t)r] * fp.inv_w, xyt[3 * (size_t)r + 1] * fp.inv_h, c, s};
#pragma unroll
        for (int d = 0; d < 4; ++d) {
            float s0, c0, s1, c1;
            sincospif(f0 * u[d], &s0, &c0);
            sincospif(f1 * u[d], &s1, &c1);
            out[d * 64] = pack_bf16(s0, c0);
            out[d * 64 + 32] = pack_bf16(s1, c1);
        }
    }
}

cudaError_t launch_features(const FeatParams& fp, const float* xyt, int n, int rows, bf16* X, cudaStream_t s) {
    if (rows <= 0) return cudaSuccess;
    return launch_next(k_features, dim3((rows + 8 * kFeatRows - 1) / (8 * kFeatRows)), 256, 0, s, fp, xyt, n, rows, X);
}

// ------------------------------------------------------ fused forward pass
// Inference of the whole network without leaving the SM: only the rays' poses come in and one float per
// ray goes out (the layer-by-layer path moves ~3.1 KB per ray through HBM).  One persistent CTA per SM
// works on two tiles of 128 rays, each with its 64 KB of activations in shared memory and its 256 TMEM
// columns:
//   warp 0       TMA producer: the weights of every layer in K chunks of 64 (32 KB), round a ring of
//                three stages, in the MMA warp's order;
//   warp 1       allocates TMEM; one thread issues the MMAs, layer by layer, tile 0 and tile 1 in turn;
//   warps 2-9    tile 0, warps 10-17 tile 1, two threads per ray (column halves): the features of a K
//                chunk straight into the A operand (the activation buffer's four 64-wide blocks are the
//                first layer's stages), each layer's epilogue (bias, bf16 rounding, GELU) from TMEM into
//                the next layer's A operand, the last one into the output layer's sums.
// The two tiles are out of step, so one's arithmetic fills the other's waits for its MMAs.  Bound by
// issuing that arithmetic: per ray 256 sincospi and 1,024 GELUs (a tanh each: 8 cycles of the SFU per
// warp).  Two CTAs per SM in step with their weights' copies before: 1.08 M rays 2.32 ms; this 0.93,
// with x and y features computed once for the beams of a pose and TMEM read ahead 0.79.  Not better:
// a stream of half-size weight stages for each tile (0.96), the tiles half a tile apart (0.99), their
// feature chunks in turn (0.82).
// Every MMA operand, rounding point and summation order matches the layer-by-layer path, so the
// predictions are bit-identical to it.  Operands K-major with the 128-byte swizzle (tc::make_desc_sw128).
// Waits are bounded as in k_gemm_tma; no role waits on a hardware barrier that another may leave.
constexpr int kFwdTile = 8 * 32;                     // threads of a tile
constexpr int kFwdThreads = 64 + 2 * kFwdTile;
constexpr int kFwdStages = 3;
constexpr uint32_t kFwdStage = kBN * tc::kKChunk * 2;     // 32 KB of weights
constexpr uint32_t kActBlock = kBM * tc::kKChunk * 2;     // 16 KB: 64 columns of a tile's activations
constexpr size_t kFwdSmem = kFwdStages * (size_t)kFwdStage + 2 * 4 * (size_t)kActBlock + 1024;

// K chunks of a layer
__host__ __device__ constexpr int layer_chunks(int l) { return (l == 0 ? kFeat : kHidden) / tc::kKChunk; }

__global__ void __launch_bounds__(kFwdThreads, 1)
k_mlp_forward(const __grid_constant__ CUtensorMap tm0, const __grid_constant__ CUtensorMap tmH, FeatParams fp,
              const float* __restrict__ xyt, int n, const float* __restrict__ params, float* __restrict__ y, unsigned* err) {
    extern __shared__ uint8_t smem_raw[];
    __shared__ __align__(8) uint64_t w_full[kFwdStages], w_empty[kFwdStages];
    __shared__ __align__(8) uint64_t a_full[2][4], a_free[2][4], acc_full[2], out_full[2], drained;
    __shared__ uint32_t tmem_base;
    __shared__ int abort_flag, n_issued, n_consumed;
    __shared__ __align__(16) float s_freq[64];
    uint8_t* smem = reinterpret_cast<uint8_t*>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    const uint32_t sW = tc::smem_addr(smem), sAct = sW + kFwdStages * kFwdStage;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    // tile i of group g is (2 i + g) * gridDim.x + blockIdx.x: few rays spread over the SMs first
    const int tiles = (n + kBM - 1) / kBM, G = gridDim.x;
    const int rounds = (tiles - (int)blockIdx.x + 2 * G - 1) / (2 * G);
    auto has_tile = [&](int i, int g) { return (2 * i + g) * G + (int)blockIdx.x < tiles; };
    if (warp == 1) tc::tmem_alloc(tc::smem_addr(&tmem_base), 512);
    if (threadIdx.x == 0) {
        for (int i = 0; i < kFwdStages; ++i) {
            tc::mbar_init(tc::smem_addr(&w_full[i]), 1);
            tc::mbar_init(tc::smem_addr(&w_empty[i]), 1);
        }
        for (int g = 0; g < 2; ++g) {
            for (int i = 0; i < 4; ++i) {
                tc::mbar_init(tc::smem_addr(&a_full[g][i]), kFwdTile / 32);
                tc::mbar_init(tc::smem_addr(&a_free[g][i]), 1);
            }
            tc::mbar_init(tc::smem_addr(&acc_full[g]), 1);
            tc::mbar_init(tc::smem_addr(&out_full[g]), kFwdTile / 64);
        }
        tc::mbar_init(tc::smem_addr(&drained), 1);
        abort_flag = 0;
        n_issued = 0;
        n_consumed = 0;
        tc::fence_mbar_init();
    }
    if (threadIdx.x < 64) s_freq[threadIdx.x] = fp.freq[threadIdx.x];
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    const uint32_t tmem = tmem_base;
    auto aborted = [&]() { return *(volatile int*)&abort_flag != 0; };
    auto give_up = [&]() {
        atomicOr(err, 16u);
        atomicExch(&abort_flag, 1);
    };
    if (warp == 0 && lane == 0) {
        // ---- producer
        tc::tma_prefetch_map(&tm0);
        tc::tma_prefetch_map(&tmH);
        int c_all = 0, st = 0, phase = 1;
        bool ok = true;
        for (int i = 0; i < rounds && ok; ++i)
            for (int lg = 0; lg < 2 * kLayers && ok; ++lg) {
                const int l = lg >> 1;
                if (!has_tile(i, lg & 1)) continue;
                for (int c = 0; c < layer_chunks(l); ++c, ++c_all) {
                    if (c_all >= kFwdStages && !tc::mbar_wait(tc::smem_addr(&w_empty[st]), phase)) {
                        give_up();
                        ok = false;
                        break;
                    }
                    const uint32_t fb = tc::smem_addr(&w_full[st]);
                    tc::mbar_arrive_expect_tx(fb, kFwdStage);
                    tc::tma_load_3d(sW + st * kFwdStage, l == 0 ? &tm0 : &tmH, c * tc::kKChunk, 0, l == 0 ? 0 : l - 1, fb);
                    if (++st == kFwdStages) {
                        st = 0;
                        phase ^= 1;
                    }
                }
            }
        n_issued = c_all;
    } else if (warp == 1 && lane == 0) {
        // ---- MMA issuer.  uses[g]: how often tile g's A blocks have been filled (all four alike)
        const uint32_t idesc = tc::make_idesc(kBM, kBN);
        const uint64_t w0 = tc::make_desc_sw128(sW), a0 = tc::make_desc_sw128(sAct);
        int c_all = 0, st = 0, phase = 0;
        unsigned uses[2] = {0, 0};
        bool ok = true;
        for (int i = 0; i < rounds && ok; ++i)
            for (int l = 0; l < kLayers && ok; ++l)
#pragma unroll
                for (int g = 0; g < 2; ++g) {
                    if (!has_tile(i, g) || !ok) continue;
                    for (int c = 0; c < layer_chunks(l); ++c) {
                        const int b = c & 3;
                        ok = tc::mbar_wait(tc::smem_addr(&a_full[g][b]), (uses[g] + (c >> 2)) & 1) &&
                             tc::mbar_wait(tc::smem_addr(&w_full[st]), phase);
                        if (!ok) break;
                        tc::fence_after_sync();
#pragma unroll
                        for (int ks = 0; ks < tc::kKChunk / 16; ++ks)
                            tc::mma_bf16(tmem + g * kBN, a0 + (uint32_t)((g * 4 + b) * (kActBlock >> 4) + ks * 2),
                                         w0 + (uint32_t)(st * (kFwdStage >> 4) + ks * 2), idesc, (c > 0 || ks > 0) ? 1u : 0u);
                        tc::mma_commit(tc::smem_addr(&w_empty[st]));
                        if (l == 0 && c < 4) tc::mma_commit(tc::smem_addr(&a_free[g][b]));
                        ++c_all;
                        if (++st == kFwdStages) {
                            st = 0;
                            phase ^= 1;
                        }
                    }
                    if (ok) tc::mma_commit(tc::smem_addr(&acc_full[g]));
                    uses[g] += layer_chunks(l) / 4;
                }
        n_consumed = c_all;
        if (!ok) {   // let what was issued end before the TMEM is freed
            give_up();
            tc::mma_commit(tc::smem_addr(&drained));
            (void)tc::mbar_wait(tc::smem_addr(&drained), 0);
        }
    } else if (warp >= 2) {
        // ---- features and epilogues
        const int g = (warp - 2) >> 3, half = ((warp - 2) >> 2) & 1;
        const int row = (warp & 3) * 32 + lane;   // TMEM lanes 32 (warp % 4) .. + 31
        uint8_t* act = smem + kFwdStages * kFwdStage + g * 4 * kActBlock + row * 128;
        const uint32_t acc = tmem + g * kBN + ((uint32_t)((warp & 3) * 32) << 16);
        const int swz = row & 7;
        const float* wout = params + kOutW;
        auto wait = [&](uint64_t* bar, uint32_t parity) {
            const bool ok = __all_sync(0xffffffffu, tc::mbar_wait(tc::smem_addr(bar), parity) && !aborted());
            if (!ok && lane == 0) give_up();
            tc::fence_after_sync();
            return ok;
        };
        bool ok = true;
        unsigned layers_done = 0;
        for (int i = 0; i < rounds && ok && has_tile(i, g); ++i) {
            const int r = ((2 * i + g) * G + (int)blockIdx.x) * kBM + row;
            const bool live = r < n;
            float u0 = 0.0f, u1 = 0.0f, u2 = 0.0f, u3 = 0.0f;
            if (live) {
                sincosf(__ldg(xyt + 3 * (size_t)r + 2), &u3, &u2);
                u0 = __ldg(xyt + 3 * (size_t)r) * fp.inv_w;
                u1 = __ldg(xyt + 3 * (size_t)r + 1) * fp.inv_h;
            }
            // features [64 c, 64 c + 64): input c / 2, frequencies 32 (c % 2) .. + 31, a thread 16 of them.
            // Where the warp's rays come from at most two positions, as 32 beams or more of a pose do, lane
            // l computes frequency l % 16 of x and y for the first (l < 16) or the second, once for them all.
            const float ax = __shfl_sync(0xffffffffu, u0, 0), ay = __shfl_sync(0xffffffffu, u1, 0);
            const float bx = __shfl_sync(0xffffffffu, u0, 31), by = __shfl_sync(0xffffffffu, u1, 31);
            const bool first = same_bits(u0, ax) && same_bits(u1, ay);
            const bool shared = __all_sync(0xffffffffu, first || (same_bits(u0, bx) && same_bits(u1, by)));
#pragma unroll 1
            for (int c = 0; c < kFeat / tc::kKChunk; ++c) {
                if (c >= 4 && !(ok = wait(&a_free[g][c & 3], i & 1))) break;
                const float* f = s_freq + (c & 1) * 32 + half * 16;
                uint8_t* out = act + (c & 3) * kActBlock;
                if (c < 4 && shared) {
                    float sn, cs;
                    sincospif(f[lane & 15] * (lane < 16 ? (c < 2 ? ax : ay) : (c < 2 ? bx : by)), &sn, &cs);
                    const uint32_t v = pack_bf16(sn, cs);   // (rows past the end take either)
                    const int from = first ? 0 : 16;
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        uint32_t o[4];
#pragma unroll
                        for (int e = 0; e < 4; ++e) o[e] = __shfl_sync(0xffffffffu, v, from + 4 * q + e);
                        *reinterpret_cast<uint4*>(out + (((half * 4 + q) ^ swz) << 4)) = make_uint4(o[0], o[1], o[2], o[3]);
                    }
                } else {
                    const float u = c < 2 ? u0 : c < 4 ? u1 : c < 6 ? u2 : u3;
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        const float4 fq = *reinterpret_cast<const float4*>(f + 4 * q);
                        uint4 o;
                        float sn, cs;
                        sincospif(fq.x * u, &sn, &cs);
                        o.x = pack_bf16(sn, cs);
                        sincospif(fq.y * u, &sn, &cs);
                        o.y = pack_bf16(sn, cs);
                        sincospif(fq.z * u, &sn, &cs);
                        o.z = pack_bf16(sn, cs);
                        sincospif(fq.w * u, &sn, &cs);
                        o.w = pack_bf16(sn, cs);
                        if (!live) o = make_uint4(0u, 0u, 0u, 0u);
                        *reinterpret_cast<uint4*>(out + (((half * 4 + q) ^ swz) << 4)) = o;
                    }
                }
                tc::fence_async_smem();
                tc::fence_before_sync();
                __syncwarp();
                if (lane == 0) tc::mbar_arrive(tc::smem_addr(&a_full[g][c & 3]));
            }
            if (!ok) break;
            // hidden layers: z = acc + b, rounded to bf16; h = bf16(GELU(z)) into the A blocks
#pragma unroll 1
            for (int l = 0; l < kLayers - 1 && ok; ++l) {
                if (!(ok = wait(&acc_full[g], layers_done++ & 1))) break;
                const float4* bias = reinterpret_cast<const float4*>(params + b_offset(l));
                const int c0 = 128 * half;
                uint32_t v[2][32];   // the next 32 columns are on their way while these are computed
                tc::tmem_ld32_issue(acc + c0, v[0]);
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    uint32_t* a = v[k & 1];
                    tc::tmem_ld32_wait(a);
                    if (k < 3) tc::tmem_ld32_issue(acc + c0 + 32 * k + 32, v[(k + 1) & 1]);
                    uint8_t* out = act + ((c0 >> 6) + (k >> 1)) * kActBlock;
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        uint32_t h[4];
#pragma unroll
                        for (int e = 0; e < 2; ++e) {
                            const int j = 8 * q + 4 * e;
                            const float4 b = __ldg(bias + (c0 + 32 * k + j) / 4);
                            const float2 z0 = unpack2(add2(pack2(__uint_as_float(a[j]), __uint_as_float(a[j + 1])), pack2(b.x, b.y)));
                            const float2 z1 = unpack2(add2(pack2(__uint_as_float(a[j + 2]), __uint_as_float(a[j + 3])), pack2(b.z, b.w)));
                            const float2 h0 = gelu(widen_bf16(pack_bf16(z0.x, z0.y))), h1 = gelu(widen_bf16(pack_bf16(z1.x, z1.y)));
                            h[2 * e] = pack_bf16(h0.x, h0.y);
                            h[2 * e + 1] = pack_bf16(h1.x, h1.y);
                        }
                        *reinterpret_cast<uint4*>(out + ((((k & 1) * 4 + q) ^ swz) << 4)) = make_uint4(h[0], h[1], h[2], h[3]);
                    }
                }
                tc::fence_async_smem();
                tc::fence_before_sync();
                __syncwarp();
                if (lane < 4) tc::mbar_arrive(tc::smem_addr(&a_full[g][lane]));
            }
            // the last layer and the output layer in k_out_layer's summation order: sums over the columns
            // j = e (mod 32) in increasing j, of which this thread has e = 16 half .. + 15, then the xor butterfly
            if (!ok || !(ok = wait(&acc_full[g], layers_done++ & 1))) break;
            const float4* bias = reinterpret_cast<const float4*>(params + b_offset(kLayers - 1));
            f32x2 part[8];
#pragma unroll
            for (int e = 0; e < 8; ++e) part[e] = 0ull;
#pragma unroll 1
            for (int cb = 16 * half; cb < kHidden; cb += 32) {
                float v[16];
                tc::tmem_ld16(acc + cb, v);
#pragma unroll
                for (int q = 0; q < 16; q += 4) {
                    const float4 b = __ldg(bias + (cb + q) / 4), w = __ldg(reinterpret_cast<const float4*>(wout + cb + q));
                    const float2 z0 = unpack2(add2(pack2(v[q], v[q + 1]), pack2(b.x, b.y)));
                    const float2 z1 = unpack2(add2(pack2(v[q + 2], v[q + 3]), pack2(b.z, b.w)));
                    const float2 h0 = gelu(widen_bf16(pack_bf16(z0.x, z0.y))), h1 = gelu(widen_bf16(pack_bf16(z1.x, z1.y)));
                    part[q / 2] = add2(part[q / 2], mul2_then(widen_bf16(pack_bf16(h0.x, h0.y)), pack2(w.x, w.y)));
                    part[q / 2 + 1] = add2(part[q / 2 + 1], mul2_then(widen_bf16(pack_bf16(h1.x, h1.y)), pack2(w.z, w.w)));
                }
            }
            float p[16];
#pragma unroll
            for (int e = 0; e < 8; ++e) {
                const float2 t = unpack2(part[e]);
                p[2 * e] = t.x;
                p[2 * e + 1] = t.y;
            }
            if (half) {   // through TMEM columns 16 .. 31, which only this thread reads
                tc::tmem_st16(acc + 16, p);
                tc::fence_before_sync();
                __syncwarp();
                if (lane == 0) tc::mbar_arrive(tc::smem_addr(&out_full[g]));
            } else {
                if (!(ok = wait(&out_full[g], i & 1))) break;
                float o[16];
                tc::tmem_ld16(acc + 16, o);
#pragma unroll
                for (int e = 0; e < 16; ++e) p[e] = __fadd_rn(p[e], o[e]);
#pragma unroll
                for (int s = 8; s; s >>= 1)
#pragma unroll
                    for (int e = 0; e < s; ++e) p[e] = __fadd_rn(p[e], p[e + s]);
                if (live) y[r] = __fadd_rn(p[0], __ldg(wout + kHidden));
            }
        }
    }
    tc::fence_before_sync();
    __syncthreads();
    if (abort_flag && threadIdx.x == 0) {
        // loads issued but never waited for are still landing in this CTA's shared memory: wait for
        // them (bounded) before the CTA exits
        for (int c = n_consumed; c < n_issued; ++c)
            (void)tc::mbar_wait(tc::smem_addr(&w_full[c % kFwdStages]), (c / kFwdStages) & 1);
    }
    __syncthreads();
    if (warp == 1) tc::tmem_dealloc(tmem, 512);
}

cudaError_t mlp_forward(const FeatParams& fp, const float* xyt, int n, const bf16* wbf, const float* params, float* y,
                        unsigned* err, cudaStream_t s) {
    if (n <= 0) return cudaSuccess;
    CUtensorMap t0, th;
    TRY(operand_map(&t0, wbf, false, kHidden, kFeat, kFeat, kHidden));
    TRY(operand_map(&th, wbf + w_offset(1), false, kHidden, kHidden, kHidden, kHidden, kLayers - 1, w_offset(2) - w_offset(1)));
    static std::atomic<unsigned long long> attr{0};
    TRY(ensure_smem_attr(k_mlp_forward, (int)kFwdSmem, attr));
    k_mlp_forward<<<std::min(152, (n - 1) / kBM + 1), kFwdThreads, kFwdSmem, s>>>(t0, th, fp, xyt, n, params, y, err);
    return cudaGetLastError();
}

// output layer: y = H . w + b (fp32)
__global__ void k_out_layer(const bf16* __restrict__ H, const float* __restrict__ params, int n, float* __restrict__ y) {
    const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (warp >= n) return;
    const bf16* h = H + (size_t)warp * kHidden;
    const float* w = params + kOutW;
    float acc = 0.0f;
    for (int j = lane; j < kHidden; j += 32) acc += __bfloat162float(h[j]) * w[j];
    for (int o = 16; o; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    if (lane == 0) y[warp] = acc + w[kHidden];
}

// --------------------------------------------------------------- training
// The output layer of a training step in one pass over its activations H and pre-activations Z, a row
// per warp: y = H . w + b (in k_out_layer's order), the Huber loss (delta 1 px) against the target and
// its gradient dy (mean over the batch), dZ = dy * w * GELU'(Z), and the block's share of the layer's
// gradients and of the loss in part[block] = {d w [256], d b, loss}.  Bound by its 3 x 512 bytes a row;
// five kernels before (loss, backward, two column sums and the output layer: 113 us for 65,536 rows,
// now 24).
constexpr int kTopBlocks = 2 * 152, kTopThreads = 512;
constexpr int kTopPart = kHidden + 2;

__global__ void __launch_bounds__(kTopThreads) k_top(const bf16* H, const bf16* Z,
                                                     const float* __restrict__ params, const float* target,
                                                     int n, bf16* __restrict__ dZ, float* __restrict__ part) {
    __shared__ float s_part[kTopThreads / 32][kTopPart];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const float* wo = params + kOutW;
    float w[8], dw[8], db = 0.0f, loss = 0.0f;
    after_previous();
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        w[i] = __ldg(wo + lane + 32 * i);
        dw[i] = 0.0f;
    }
    const float b = __ldg(wo + kHidden);
    const int warps = gridDim.x * (kTopThreads / 32);
#pragma unroll 2
    for (int r = blockIdx.x * (kTopThreads / 32) + warp; r < n; r += warps) {
        const size_t base = (size_t)r * kHidden + lane;
        float h[8], z[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            h[i] = __bfloat162float(H[base + 32 * i]);
            z[i] = __bfloat162float(Z[base + 32 * i]);
        }
        const float t = target[r];
        float acc = 0.0f;
#pragma unroll
        for (int i = 0; i < 8; ++i) acc += h[i] * w[i];
        for (int o = 16; o; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
        const float e = (acc + b) - t, ae = fabsf(e);
        const float dy = (ae <= 1.0f ? e : copysignf(1.0f, e)) / (float)n;
        loss += ae <= 1.0f ? 0.5f * e * e : ae - 0.5f;
        db += dy;
#pragma unroll
        for (int i = 0; i < 8; i += 2) {
            const float2 d = unpack2(mul2(mul2(both(dy), pack2(w[i], w[i + 1])), gelu_grad(pack2(z[i], z[i + 1]))));
            dZ[base + 32 * i] = __float2bfloat16_rn(d.x);
            dZ[base + 32 * i + 32] = __float2bfloat16_rn(d.y);
        }
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            dw[i] += dy * h[i];
        }
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) s_part[warp][lane + 32 * i] = dw[i];
    if (lane == 0) {
        s_part[warp][kHidden] = db;
        s_part[warp][kHidden + 1] = loss;
    }
    __syncthreads();
    for (int j = threadIdx.x; j < kTopPart; j += kTopThreads) {
        float sum = 0.0f;
        for (int k = 0; k < kTopThreads / 32; ++k) sum += s_part[k][j];
        part[(size_t)blockIdx.x * kTopPart + j] = sum;
    }
}

// The gradients from their partial sums, always added in the same order: the hidden layers' from the
// K splits of the weight-gradient GEMMs (part[z][kOutW], the flat parameter layout), the output
// layer's and the loss from k_top's blocks.  A run repeats bit for bit; the sums were atomic before.
// Then the parameter's step, where there is one: Adam (bias-corrected), fp32 master weights; refreshes the
// bf16 copies the GEMMs read.
struct AdamArgs {
    float *p, *m, *v;   // p null: gradients only
    bf16* wbf;
    float lr, b1, b2, eps, c1, c2;
};

__device__ __forceinline__ void adam(const AdamArgs& A, size_t i, float gi) {
    const float mi = A.b1 * A.m[i] + (1.0f - A.b1) * gi;
    const float vi = A.b2 * A.v[i] + (1.0f - A.b2) * gi * gi;
    A.m[i] = mi;
    A.v[i] = vi;
    const float pi = A.p[i] - A.lr * (mi * A.c1) / (sqrtf(vi * A.c2) + A.eps);
    A.p[i] = pi;
    A.wbf[i] = __float2bfloat16_rn(pi);
}

__global__ void __launch_bounds__(256) k_reduce_grads(const float* part, int splits,
                                                      const float* top, float* __restrict__ grads,
                                                      float* __restrict__ loss, AdamArgs A) {
    constexpr unsigned kHiddenBlocks = (unsigned)(kOutW / 256);
    after_previous();
    if (blockIdx.x < kHiddenBlocks) {
        const size_t i = (size_t)blockIdx.x * 256 + threadIdx.x;
        float sum = 0.0f;
#pragma unroll 16
        for (int z = 0; z < splits; ++z) sum += part[(size_t)z * kOutW + i];
        grads[i] = sum;
        if (A.p) adam(A, i, sum);
        return;
    }
    const int j = (int)(blockIdx.x - kHiddenBlocks) * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (j >= kTopPart) return;
    float sum = 0.0f;
    for (int k = lane; k < kTopBlocks; k += 32) sum += top[(size_t)k * kTopPart + j];
    for (int o = 16; o; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
    if (lane != 0) return;
    if (j <= kHidden) {
        grads[kOutW + j] = sum;
        if (A.p) adam(A, kOutW + j, sum);
    } else {
        *loss = sum;
    }
}

__global__ void k_to_bf16(const float* __restrict__ src, bf16* __restrict__ dst, size_t n) {
    size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) dst[i] = __float2bfloat16_rn(src[i]);
}

__device__ __forceinline__ uint32_t hash32(uint32_t x) {
    x ^= x >> 16; x *= 0x7feb352du; x ^= x >> 15; x *= 0x846ca68bu; x ^= x >> 16;
    return x;
}
__device__ __forceinline__ float u01(uint32_t a, uint32_t b) {
    return (hash32(a * 0x9e3779b9u ^ hash32(b)) >> 8) * (1.0f / 16777216.0f);
}

// uniform(-1/sqrt(fan_in), 1/sqrt(fan_in)) weights, zero biases, output bias = init_bias
__global__ void k_init_params(float* __restrict__ p, uint32_t seed, float init_bias) {
    size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= kParamCount) return;
    float val = 0.0f;
    for (int l = 0; l < kLayers; ++l) {
        size_t w0 = w_offset(l), nw = (size_t)kHidden * layer_in(l);
        if (i >= w0 && i < w0 + nw) val = (2.0f * u01(seed, (uint32_t)i) - 1.0f) * rsqrtf((float)layer_in(l)) * 1.7f;
    }
    if (i >= kOutW && i < kOutW + kHidden) val = (2.0f * u01(seed, (uint32_t)i) - 1.0f) * rsqrtf((float)kHidden);
    if (i == kOutW + kHidden) val = init_bias;
    p[i] = val;
}

// the reference's range: from (x0, y0) to the corner of cell (px, py)
__device__ __forceinline__ float corner_range(unsigned px, unsigned py, float x0, float y0) {
    const float xd = __fsub_rn(__int2float_rn((int)px), x0), yd = __fsub_rn(__int2float_rn((int)py), y0);
    return __fsqrt_rn(__fadd_rn(__fmul_rn(xd, xd), __fmul_rn(yd, yd)));
}

// ---------------------------------------------------- rays from the marcher
// The exact march (RangeLib.h:927-962) also reporting t at the hit step;
// t = max_range when the ray leaves the map or runs out of range.
__device__ float march_t(const MapDev& m, float mr, float x0, float y0, float c, float s, float* range) {
    const unsigned W = (unsigned)m.W, H = (unsigned)m.H;
    float t = 0.0f, at = mr;
    unsigned px = 0, py = 0;
    bool hit = false;
    if (m.step) {   // NaN on occupied cells, +inf off the grid (MapDev::step): one comparison ends the march
        while (t < mr) {
            at = t;
            px = (unsigned)__float2int_rz(__fadd_rn(x0, __fmul_rn(c, t)));
            py = (unsigned)__float2int_rz(__fadd_rn(y0, __fmul_rn(s, t)));
            t = __fadd_rn(t, __ldg(m.step + (min(px, W) * (H + 1u) + min(py, H))));
        }
        hit = isnan(t);
    } else {
        while (t < mr) {
            at = t;
            px = (unsigned)__float2int_rz(__fadd_rn(x0, __fmul_rn(c, t)));
            py = (unsigned)__float2int_rz(__fadd_rn(y0, __fmul_rn(s, t)));
            if (px >= W || py >= H) break;
            const float d = __ldg(m.dt + (size_t)px * m.H + py);
            if (d <= 0.0f) {
                hit = true;
                break;
            }
            t = __fadd_rn(t, fmaxf(__fmul_rn(d, 0.999f), 1.0f));
        }
    }
    if (!hit) {
        *range = mr;
        return mr;
    }
    *range = corner_range(px, py, x0, y0);
    return at;
}

// random free-cell poses, uniform heading; xyt (grid frame), t target, exact range
__global__ void k_sample_rays(MapDev m, float mr, const uint32_t* __restrict__ free_cells, uint32_t n_free,
                              uint32_t seed, long long base, int n, float* __restrict__ xyt, float* __restrict__ t,
                              float* __restrict__ range) {
    int r = blockIdx.x * blockDim.x + threadIdx.x;
    after_previous();
    if (r >= n) return;
    const uint32_t id = (uint32_t)(base + r);
    const uint32_t cell = free_cells[hash32(id ^ hash32(seed)) % n_free];
    const int cx = (int)(cell / (uint32_t)m.H), cy = (int)(cell - (uint32_t)cx * (uint32_t)m.H);
    const float x = (float)cx + u01(id, seed ^ 0x1u), y = (float)cy + u01(id, seed ^ 0x2u);
    const float th = 6.2831853f * u01(id, seed ^ 0x3u);
    xyt[3 * (size_t)r] = x;
    xyt[3 * (size_t)r + 1] = y;
    xyt[3 * (size_t)r + 2] = th;
    float s, c, rg;
    rlc_trig::sincos_cr(th, &s, &c);   // the exact path's cos/sin
    t[r] = march_t(m, mr, x, y, c, s, &rg);
    if (range) range[r] = rg;
}

__global__ void k_free_flags(const uint64_t* __restrict__ bits, int W, int H, int TY, uint32_t* __restrict__ f) {
    long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= (long long)W * H) return;
    int x = (int)(i / H), y = (int)(i - (long long)x * H);
    uint64_t w = bits[(size_t)(x >> 3) * TY + (y >> 3)];
    f[i] = ((w >> (((x & 7) << 3) | (y & 7))) & 1ull) ? 0u : 1u;
}

__global__ void k_compact_free(const uint32_t* __restrict__ f, const uint32_t* __restrict__ pos, long long n,
                               uint32_t* __restrict__ out) {
    long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n && f[i]) out[pos[i]] = (uint32_t)i;
}

// ------------------------------------------------------- learned inference
__device__ __forceinline__ bool occ_cell(const MapDev& m, int x, int y) {
    if ((unsigned)x >= (unsigned)m.W || (unsigned)y >= (unsigned)m.H) return false;
    uint64_t w = __ldg(m.bits + (size_t)(x >> 3) * m.tiles_y + (y >> 3));
    return (w >> (((x & 7) << 3) | (y & 7))) & 1ull;
}

// A ray whose predicted hit cell is occupied and the cell a step before it free is accepted: the range to
// that cell's corner.  The block's other rays are collected with their direction and marched exactly, 32
// at a time per warp as warps come free (lanes taking rays one by one: 98 us).  (Two passes with a list in memory, and the march's two tests a
// step: 103 us for 1.08 M rays of which all are recast, now 86.)
constexpr int kResolveRays = 1024, kResolveThreads = 256;

__global__ void __launch_bounds__(kResolveThreads) k_resolve(MapDev m, float mr, const float* __restrict__ xyt,
                                                             const float* __restrict__ pred, int n, float scale,
                                                             float* __restrict__ outs, uint8_t* __restrict__ accepted,
                                                             int* __restrict__ n_recast) {
    __shared__ float4 s_ray[kResolveRays];
    __shared__ unsigned short s_id[kResolveRays];
    __shared__ int s_count, s_next;
    if (threadIdx.x == 0) s_count = s_next = 0;
    __syncthreads();
    const int lane = threadIdx.x & 31;
    const long long base = (long long)blockIdx.x * kResolveRays;
#pragma unroll
    for (int j = 0; j < kResolveRays / kResolveThreads; ++j) {
        const int id = j * kResolveThreads + (int)threadIdx.x;
        const long long r = base + id;
        bool recast = false;
        float x0 = 0.0f, y0 = 0.0f, s = 0.0f, c = 0.0f;
        if (r < n) {
            x0 = __ldg(xyt + 3 * r);
            y0 = __ldg(xyt + 3 * r + 1);
            rlc_trig::sincos_cr(__ldg(xyt + 3 * r + 2), &s, &c);
            const float t = __ldg(pred + r);
            bool ok = false;
            if (t > 1.0f && t < 0.999f * mr && isfinite(t)) {
                const int hx = __float2int_rz(x0 + c * t), hy = __float2int_rz(y0 + s * t);
                const int bx = __float2int_rz(x0 + c * (t - 1.0f)), by = __float2int_rz(y0 + s * (t - 1.0f));
                if (occ_cell(m, hx, hy) && !occ_cell(m, bx, by)) {
                    outs[r] = __fmul_rn(corner_range((unsigned)hx, (unsigned)hy, x0, y0), scale);
                    ok = true;
                }
            }
            if (accepted) accepted[r] = ok ? 1 : 0;
            recast = !ok;
        }
        const unsigned who = __ballot_sync(0xffffffffu, recast);
        if (who) {
            int slot = 0;
            if (lane == 0) slot = atomicAdd(&s_count, __popc(who));
            slot = __shfl_sync(0xffffffffu, slot, 0) + __popc(who & ((1u << lane) - 1u));
            if (recast) {
                s_ray[slot] = make_float4(x0, y0, c, s);
                s_id[slot] = (unsigned short)id;
            }
        }
    }
    __syncthreads();
    const int count = s_count;
    if (threadIdx.x == 0 && count) atomicAdd(n_recast, count);
    for (;;) {
        int i = 0;
        if (lane == 0) i = atomicAdd(&s_next, 32);
        i = __shfl_sync(0xffffffffu, i, 0);
        if (i >= count) break;
        i += lane;
        if (i < count) {
            const float4 q = s_ray[i];
            float rg;
            march_t(m, mr, q.x, q.y, q.z, q.w, &rg);
            outs[base + s_id[i]] = __fmul_rn(rg, scale);
        }
    }
}



// world-frame particles x beams -> grid-frame rays (RangeLib.h:482-520)
__global__ void k_world_rays(WorldDev w, const float* __restrict__ ins, const float* __restrict__ angles, int n,
                             int na, float* __restrict__ xyt) {
    long long g = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (g >= (long long)n * na) return;
    int i = (int)(g / na), a = (int)(g - (long long)i * na);
    float x = __fmul_rn(__fsub_rn(ins[3 * (size_t)i], w.ox), w.inv_s);
    float y = __fmul_rn(__fsub_rn(ins[3 * (size_t)i + 1], w.oy), w.inv_s);
    float tmp = x;
    x = __fsub_rn(__fmul_rn(w.ca, x), __fmul_rn(w.sa, y));
    y = __fadd_rn(__fmul_rn(w.sa, tmp), __fmul_rn(w.ca, y));
    const float th = __fsub_rn(__fadd_rn(-ins[3 * (size_t)i + 2], w.rc), angles[a]);
    xyt[3 * g] = y;   // calc_range(y, x, theta)
    xyt[3 * g + 1] = x;
    xyt[3 * g + 2] = th;
}

inline unsigned blocks_for(long long n, int b) { return (unsigned)((n + b - 1) / b); }

}  // namespace

// ================================================================ host side
struct LearnedModel {
    MapDev map{};
    WorldDev world{};
    float mr = 0.0f;
    FeatParams fp{};
    float* params = nullptr;   // fp32 master [kParamCount]
    float* adam_m = nullptr;
    float* adam_v = nullptr;
    float* grads = nullptr;
    bf16* wbf = nullptr;       // bf16 copy of params (weights used by the GEMMs)
    unsigned* err = nullptr;   // {bits raised by waits that ran out since they were last taken, recast rays of a query}
    long long adam_t = 0;
    // work buffers for a chunk of `cap` rays
    int cap = 0;
    bf16* X = nullptr;                 // [cap x 512]
    bf16* Z[kLayers] = {};             // pre-activations [cap x 256]
    bf16* Hh[kLayers] = {};            // activations
    bf16* dZ[2] = {};                  // ping-pong gradients
    float* wpart = nullptr;            // partial gradients of the hidden layers [kMaxSplits][kOutW]
    float* tpart = nullptr;            // and of the output layer [kTopBlocks][kTopPart]
    float* y = nullptr;
    float* loss = nullptr;             // of the last kLossSlots steps
    float* ray_xyt = nullptr;          // the rays of a training step [cap x 3] and their targets
    float* ray_t = nullptr;
    uint32_t* free_cells = nullptr;
    uint32_t n_free = 0;
    // query buffers (rays of one learned call)
    long long qcap = 0;
    float* q_xyt = nullptr;
    float* q_pred = nullptr;

    cudaError_t ensure_query(long long rays) {
        if (rays <= qcap) return cudaSuccess;
        cudaFree(q_xyt); cudaFree(q_pred);
        q_xyt = q_pred = nullptr; qcap = 0;
        TRY(cudaMalloc(&q_xyt, (size_t)rays * 3 * sizeof(float)));
        TRY(cudaMalloc(&q_pred, (size_t)rays * sizeof(float)));
        qcap = rays;
        return cudaSuccess;
    }

    void free_work() {
        cudaFree(X);
        for (int l = 0; l < kLayers; ++l) { cudaFree(Z[l]); cudaFree(Hh[l]); Z[l] = Hh[l] = nullptr; }
        cudaFree(dZ[0]); cudaFree(dZ[1]);
        cudaFree(wpart); cudaFree(tpart);
        cudaFree(y); cudaFree(loss); cudaFree(ray_xyt); cudaFree(ray_t);
        X = nullptr; dZ[0] = dZ[1] = nullptr; y = loss = ray_xyt = ray_t = wpart = tpart = nullptr;
        cap = 0;
    }
    ~LearnedModel() {
        free_work();
        cudaFree(params); cudaFree(adam_m); cudaFree(adam_v); cudaFree(grads); cudaFree(wbf); cudaFree(err);
        cudaFree(free_cells);
        cudaFree(q_xyt); cudaFree(q_pred);
    }
    cudaError_t ensure(int rows) {
        rows = (rows + kBM - 1) / kBM * kBM;
        if (rows <= cap) return cudaSuccess;
        free_work();
        TRY(cudaMalloc(&X, (size_t)rows * kFeat * sizeof(bf16)));
        for (int l = 0; l < kLayers; ++l) {
            TRY(cudaMalloc(&Z[l], (size_t)rows * kHidden * sizeof(bf16)));
            TRY(cudaMalloc(&Hh[l], (size_t)rows * kHidden * sizeof(bf16)));
        }
        TRY(cudaMalloc(&dZ[0], (size_t)rows * kHidden * sizeof(bf16)));
        TRY(cudaMalloc(&dZ[1], (size_t)rows * kHidden * sizeof(bf16)));
        TRY(cudaMalloc(&wpart, (size_t)std::min(kMaxSplits, std::max(1, rows / 256)) * kOutW * sizeof(float)));
        TRY(cudaMalloc(&tpart, (size_t)kTopBlocks * kTopPart * sizeof(float)));
        TRY(cudaMalloc(&y, (size_t)rows * sizeof(float)));
        TRY(cudaMalloc(&loss, (kLossSlots + 1) * sizeof(float)));
        TRY(cudaMalloc(&ray_xyt, (size_t)rows * 3 * sizeof(float)));
        TRY(cudaMalloc(&ray_t, (size_t)rows * sizeof(float)));
        cap = rows;
        return cudaSuccess;
    }

    // K split of the weight-gradient GEMMs: equal chunks of >= 256 rows, at most kMaxSplits.  The split
    // is part of the result: where a gradient nearly cancels, Adam turns another order of its sum into
    // another step.
    static constexpr int kMaxSplits = 64;
    static constexpr int kLossSlots = 20;
    static int split_k(int rows) {
        int sp = rows;
        for (int parts = kMaxSplits; parts > 1; parts >>= 1)
            if (rows % (parts * 256) == 0) { sp = rows / parts; break; }
        return sp;
    }

    // Waits for the stream's work and takes the error word: words[0] the bits, which are cleared (a wait that
    // ran out spoils what was under way, not the calls after), words[1] the count.
    cudaError_t take(unsigned* words, cudaStream_t s) {
        TRY(cudaMemcpyAsync(words, err, 2 * sizeof(unsigned), cudaMemcpyDeviceToHost, s));
        TRY(cudaStreamSynchronize(s));
        return words[0] ? cudaMemsetAsync(err, 0, sizeof(unsigned), s) : cudaSuccess;
    }

    GemmArgs base_args() const {
        GemmArgs g{};
        g.err = err;
        return g;
    }

    // forward over `rows` rays whose features are in X; predictions in y
    cudaError_t forward(int rows, cudaStream_t s) {
        TRY(forward_hidden(rows, s));
        k_out_layer<<<blocks_for((long long)rows * 32, 256), 256, 0, s>>>(Hh[kLayers - 1], params, rows, y);
        return cudaGetLastError();
    }

    cudaError_t forward_hidden(int rows, cudaStream_t s) {
        LayerArgs g{};
        g.rows = rows;
        g.err = err;
        for (int l = 0; l < kLayers; ++l) {
            g.bias = params + b_offset(l); g.Zout = Z[l]; g.Hout = Hh[l];
            if (l == 0) TRY((layer<128, kFeat, true>(X, wbf, g, s)));
            else TRY((layer<256, kHidden, true>(Hh[l - 1], wbf + w_offset(l), g, s)));
        }
        return cudaSuccess;
    }

    // the output layer's forward and the whole backward pass of `rows` rays (features in X, the hidden
    // layers' forward state in Z/Hh, targets t); gradients into grads, the summed loss into loss[slot], and
    // the step on them
    cudaError_t backward(const float* t, int rows, int slot, const AdamArgs& adam, cudaStream_t s) {
        TRY(launch_next(k_top, dim3(kTopBlocks), kTopThreads, 0, s, Hh[kLayers - 1], Z[kLayers - 1], params, t, rows, dZ[0], tpart));
        int cur = 0;
        const int ks = split_k(rows);
        for (int l = kLayers - 1; l >= 0; --l) {
            // weight gradient: dW [out x in] = dZ^T . input (K = rows, split across CTAs), both operands as
            // they lie; the bias gradient on the way
            GemmArgs gw = base_args();
            gw.A = dZ[cur]; gw.lda = kHidden; gw.a_t = 1;                        // dZ[k=row][m=out]
            gw.B = l == 0 ? X : Hh[l - 1]; gw.ldb = layer_in(l); gw.b_t = 1;      // input[k=row][n=in]
            gw.M = kHidden; gw.N = layer_in(l); gw.K = rows;
            gw.ksplit = ks;
            gw.ldc = layer_in(l); gw.C = wpart + w_offset(l); gw.part_stride = kOutW;
            gw.k_sums = wpart + b_offset(l);
            TRY(gemm(gw, s));
            if (l == 0) break;
            // input gradient: dH = dZ . W, then times GELU'(Z[l-1])
            LayerArgs gx{};
            gx.rows = rows; gx.Zin = Z[l - 1]; gx.dZ = dZ[cur ^ 1]; gx.err = err;
            TRY((layer<256, kHidden, false>(dZ[cur], wbf + w_offset(l), gx, s)));
            cur ^= 1;
        }
        return launch_next(k_reduce_grads, dim3((unsigned)(kOutW / 256) + blocks_for(kTopPart, 8)), 256, 0, s, wpart, rows / ks,
                           tpart, grads, loss + slot, adam);
    }

    cudaError_t features(const float* xyt, int n, cudaStream_t s) {
        return launch_features(fp, xyt, n, (n + kBM - 1) / kBM * kBM, X, s);
    }

    AdamArgs adam_step(float lr) {
        ++adam_t;
        const float b1 = 0.9f, b2 = 0.999f;
        const float c1 = 1.0f / (1.0f - powf(b1, (float)adam_t)), c2 = 1.0f / (1.0f - powf(b2, (float)adam_t));
        return AdamArgs{params, adam_m, adam_v, wbf, lr, b1, b2, 1e-8f, c1, c2};
    }
};

}  // namespace rlc

// ======================================================================= ABI
using namespace rlc;

struct rlc_learned {
    LearnedModel m;
};

namespace {
char g_msg[512];
constexpr const char* kTimedOut = "tensor-core GEMM timed out waiting for its MMAs";
int lfail(int code, const char* what, cudaError_t e = cudaSuccess) {
    if (e != cudaSuccess) snprintf(g_msg, sizeof(g_msg), "%s: %s", what, cudaGetErrorString(e));
    else snprintf(g_msg, sizeof(g_msg), "%s", what);
    return set_last_error(code, g_msg);
}
#define LTRY(expr, what) do { cudaError_t _e = (expr); if (_e != cudaSuccess) return lfail(RLC_ERR_CUDA, what, _e); } while (0)
}  // namespace

extern "C" {

int rlc_learned_create(const rlc_method* rm, unsigned seed, rlc_learned** out) {
    if (!out) return lfail(RLC_ERR_ARG, "null output handle");
    *out = nullptr;
    MapDev map;
    WorldDev world;
    float mr;
    if (int rc = method_map_view(rm, &map, &world, &mr)) return rc;
    rlc_learned* L = new rlc_learned();
    LearnedModel& M = L->m;
    M.map = map;
    M.world = world;
    M.mr = mr;
    M.fp.inv_w = 1.0f / (float)map.W;
    M.fp.inv_h = 1.0f / (float)map.H;
    const double fmax = std::max(2.0, 0.5 * std::max(map.W, map.H));
    for (int k = 0; k < 64; ++k) M.fp.freq[k] = (float)std::pow(fmax, k / 63.0);
    cudaError_t e = cudaSuccess;
    if (e == cudaSuccess) e = cudaMalloc(&M.params, kParamCount * sizeof(float));
    if (e == cudaSuccess) e = cudaMalloc(&M.adam_m, kParamCount * sizeof(float));
    if (e == cudaSuccess) e = cudaMalloc(&M.adam_v, kParamCount * sizeof(float));
    if (e == cudaSuccess) e = cudaMalloc(&M.grads, kParamCount * sizeof(float));
    if (e == cudaSuccess) e = cudaMalloc(&M.wbf, kParamCount * sizeof(bf16));
    if (e == cudaSuccess) e = cudaMalloc(&M.err, 2 * sizeof(unsigned));
    if (e == cudaSuccess) e = cudaMemset(M.err, 0, 2 * sizeof(unsigned));
    if (e == cudaSuccess) e = cudaMemset(M.adam_m, 0, kParamCount * sizeof(float));
    if (e == cudaSuccess) e = cudaMemset(M.adam_v, 0, kParamCount * sizeof(float));
    if (e == cudaSuccess) {
        k_init_params<<<blocks_for((long long)kParamCount, 256), 256>>>(M.params, seed, 0.25f * mr);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) {
        k_to_bf16<<<blocks_for((long long)kParamCount, 256), 256>>>(M.params, M.wbf, kParamCount);
        e = cudaGetLastError();
    }
    // free cells of the map, for sampling training rays
    if (e == cudaSuccess) {
        const long long n = (long long)map.W * map.H;
        uint32_t *f = nullptr, *pos = nullptr;
        e = cudaMalloc(&f, (n + 1) * sizeof(uint32_t));
        if (e == cudaSuccess) e = cudaMalloc(&pos, (n + 1) * sizeof(uint32_t));
        if (e == cudaSuccess) {
            k_free_flags<<<blocks_for(n, 256), 256>>>(map.bits, map.W, map.H, map.tiles_y, f);
            e = cudaGetLastError();
        }
        if (e == cudaSuccess) e = scan_exclusive_u32(f, pos, (size_t)n, 0);
        if (e == cudaSuccess) e = cudaMemcpy(&M.n_free, pos + n, sizeof(uint32_t), cudaMemcpyDeviceToHost);
        if (e == cudaSuccess) e = cudaMalloc(&M.free_cells, (size_t)(M.n_free ? M.n_free : 1) * sizeof(uint32_t));
        if (e == cudaSuccess) {
            k_compact_free<<<blocks_for(n, 256), 256>>>(f, pos, n, M.free_cells);
            e = cudaGetLastError();
        }
        if (e == cudaSuccess) e = cudaDeviceSynchronize();
        cudaFree(f);
        cudaFree(pos);
    }
    if (e != cudaSuccess) {
        delete L;
        return lfail(RLC_ERR_CUDA, "learned model setup", e);
    }
    if (M.n_free == 0) {
        delete L;
        return lfail(RLC_ERR_ARG, "the map has no free cell to sample rays from");
    }
    *out = L;
    return RLC_OK;
}

int rlc_learned_destroy(rlc_learned* L) {
    delete L;
    return RLC_OK;
}

int64_t rlc_learned_param_count(void) { return (int64_t)kParamCount; }

int rlc_learned_get_params(rlc_learned* L, float* host_params) {
    if (!L || !host_params) return lfail(RLC_ERR_ARG, "null argument");
    LTRY(cudaMemcpy(host_params, L->m.params, kParamCount * sizeof(float), cudaMemcpyDeviceToHost), "get params");
    return RLC_OK;
}

int rlc_learned_set_params(rlc_learned* L, const float* host_params) {
    if (!L || !host_params) return lfail(RLC_ERR_ARG, "null argument");
    LTRY(cudaMemcpy(L->m.params, host_params, kParamCount * sizeof(float), cudaMemcpyHostToDevice), "set params");
    k_to_bf16<<<blocks_for((long long)kParamCount, 256), 256>>>(L->m.params, L->m.wbf, kParamCount);
    LTRY(cudaGetLastError(), "set params");
    LTRY(cudaMemset(L->m.adam_m, 0, kParamCount * sizeof(float)), "set params");
    LTRY(cudaMemset(L->m.adam_v, 0, kParamCount * sizeof(float)), "set params");
    L->m.adam_t = 0;
    return RLC_OK;
}

// Sample rays from the map's free cells with the exact marcher (device buffers, n rays).
int rlc_learned_sample_rays(rlc_learned* L, long long first_id, unsigned seed, int n, float* d_xyt, float* d_t,
                            float* d_range, void* stream) {
    if (!L || n < 0 || (n > 0 && (!d_xyt || !d_t))) return lfail(RLC_ERR_ARG, "bad argument");
    if (n == 0) return RLC_OK;
    LearnedModel& M = L->m;
    k_sample_rays<<<blocks_for(n, 256), 256, 0, (cudaStream_t)stream>>>(M.map, M.mr, M.free_cells, M.n_free, seed,
                                                                        first_id, n, d_xyt, d_t, d_range);
    LTRY(cudaGetLastError(), "sample rays");
    return RLC_OK;
}

// Forward only: predicted t for n grid-frame rays (device buffers).
int rlc_learned_predict(rlc_learned* L, const float* d_xyt, int n, float* d_pred, void* stream) {
    if (!L || n < 0 || (n > 0 && (!d_xyt || !d_pred))) return lfail(RLC_ERR_ARG, "bad argument");
    LearnedModel& M = L->m;
    LTRY(mlp_forward(M.fp, d_xyt, n, M.wbf, M.params, d_pred, M.err, (cudaStream_t)stream), "fused forward");
    return RLC_OK;
}

// The same predictions through the training path's layer-by-layer GEMMs (test reference).
int rlc_learned_predict_layered(rlc_learned* L, const float* d_xyt, int n, float* d_pred, void* stream) {
    if (!L || n < 0 || (n > 0 && (!d_xyt || !d_pred))) return lfail(RLC_ERR_ARG, "bad argument");
    LearnedModel& M = L->m;
    cudaStream_t s = (cudaStream_t)stream;
    const int chunk = 262144;
    LTRY(M.ensure(std::min(n, chunk)), "predict buffers");
    for (int off = 0; off < n; off += chunk) {
        const int cnt = std::min(chunk, n - off);
        const int rows = (cnt + kBM - 1) / kBM * kBM;
        LTRY(M.features(d_xyt + 3 * (size_t)off, cnt, s), "features");
        LTRY(M.forward(rows, s), "forward");
        LTRY(cudaMemcpyAsync(d_pred + off, M.y, cnt * sizeof(float), cudaMemcpyDeviceToDevice, s), "predict");
    }
    return RLC_OK;
}

// Test hook: the bf16 features of n grid-frame rays into d_out [n x 512] (device).
int rlc_learned_features(rlc_learned* L, const float* d_xyt, int n, void* d_out) {
    if (!L || n <= 0 || !d_xyt || !d_out) return lfail(RLC_ERR_ARG, "bad argument");
    LTRY(launch_features(L->m.fp, d_xyt, n, n, (bf16*)d_out, 0), "features");
    LTRY(cudaDeviceSynchronize(), "features");
    return RLC_OK;
}

// One forward + backward over n rays (device buffers) without an update:
// host_grads receives the parameter gradients of the mean Huber loss.
int rlc_learned_gradients(rlc_learned* L, const float* d_xyt, const float* d_t, int n, float* host_grads,
                          float* host_loss) {
    if (!L || n <= 0 || !d_xyt || !d_t) return lfail(RLC_ERR_ARG, "bad argument");
    if (n % kBM) return lfail(RLC_ERR_ARG, "gradients take a multiple of 128 rays");
    LearnedModel& M = L->m;
    LTRY(M.ensure(n), "gradient buffers");
    LTRY(M.features(d_xyt, n, 0), "features");
    LTRY(M.forward_hidden(n, 0), "forward");
    LTRY(M.backward(d_t, n, 0, AdamArgs{}, 0), "backward");
    unsigned words[2];
    LTRY(M.take(words, 0), "gradients");
    if (words[0]) return lfail(RLC_ERR_CUDA, kTimedOut);
    if (host_grads) LTRY(cudaMemcpy(host_grads, M.grads, kParamCount * sizeof(float), cudaMemcpyDeviceToHost), "grads");
    if (host_loss) {
        float l = 0.0f;
        LTRY(cudaMemcpy(&l, M.loss, sizeof(float), cudaMemcpyDeviceToHost), "loss");
        *host_loss = l / (float)n;
    }
    return RLC_OK;
}

// Train on rays drawn by the exact marcher: `steps` Adam steps of `batch` rays
// (a multiple of 128), cosine-decayed learning rate from lr.  *final_loss gets
// the mean loss of the last 20 steps.
int rlc_learned_train(rlc_learned* L, int steps, int batch, float lr, unsigned seed, float* final_loss,
                      void* stream) {
    if (!L || steps < 0 || batch <= 0 || batch % kBM) return lfail(RLC_ERR_ARG, "batch must be a positive multiple of 128");
    LearnedModel& M = L->m;
    cudaStream_t s = (cudaStream_t)stream;
    LTRY(M.ensure(batch), "train buffers");
    float *xyt = M.ray_xyt, *tt = M.ray_t;   // kept: two allocations and frees a call cost up to 150 us
    cudaError_t e = cudaSuccess;
    float loss_acc = 0.0f;
    int loss_n = 0;
    for (int st = 0; st < steps && e == cudaSuccess; ++st) {
        e = launch_next(k_sample_rays, dim3(blocks_for(batch, 256)), 256, 0, s, M.map, M.mr, M.free_cells, M.n_free, seed,
                        (long long)st * batch, batch, xyt, tt, nullptr);
        if (e == cudaSuccess) e = M.features(xyt, batch, s);
        if (e == cudaSuccess) e = M.forward_hidden(batch, s);
        const int slot = st - (steps - LearnedModel::kLossSlots);   // the last steps' losses are reported
        const float cosine = 0.5f * (1.0f + cosf(3.14159265f * (float)st / (float)(steps > 1 ? steps : 1)));
        if (e == cudaSuccess)
            e = M.backward(tt, batch, slot >= 0 ? slot : LearnedModel::kLossSlots, M.adam_step(lr * (0.05f + 0.95f * cosine)), s);
    }
    float losses[LearnedModel::kLossSlots] = {};
    if (e == cudaSuccess && steps > 0)
        e = cudaMemcpyAsync(losses, M.loss, sizeof(losses), cudaMemcpyDeviceToHost, s);
    unsigned words[2] = {};
    if (e == cudaSuccess) e = M.take(words, s);
    if (e != cudaSuccess) return lfail(RLC_ERR_CUDA, "training", e);
    if (words[0]) return lfail(RLC_ERR_CUDA, kTimedOut);
    for (int st = std::max(0, steps - LearnedModel::kLossSlots); st < steps; ++st) {
        loss_acc += losses[st - (steps - LearnedModel::kLossSlots)] / (float)batch;
        ++loss_n;
    }
    if (final_loss) *final_loss = loss_n ? loss_acc / loss_n : 0.0f;
    return RLC_OK;
}

// Learned calc_range_repeat_angles (world frame, device buffers): predicted
// hit cells that pass the check give the reference's corner distance, the
// rest are recast exactly.  accepted (optional) marks accepted rays; *n_recast
// gets the number of recast rays.
int rlc_learned_calc_range_repeat_angles(rlc_learned* L, const float* d_ins, const float* d_angles, float* d_outs,
                                         int n, int na, uint8_t* d_accepted, int64_t* n_recast, void* stream) {
    if (!L || n < 0 || na < 0) return lfail(RLC_ERR_ARG, "bad argument");
    const long long rays = (long long)n * na;
    if (rays == 0) return RLC_OK;
    if (!d_ins || !d_angles || !d_outs) return lfail(RLC_ERR_ARG, "null array");
    if (rays > (1ll << 31) - 1) return lfail(RLC_ERR_ARG, "too many rays");
    LearnedModel& M = L->m;
    cudaStream_t s = (cudaStream_t)stream;
    LTRY(M.ensure_query(rays), "learned query buffers");
    float* xyt = M.q_xyt;
    float* pred = M.q_pred;
    int* cnt = (int*)(M.err + 1);
    cudaError_t e = cudaMemsetAsync(cnt, 0, sizeof(int), s);
    if (e == cudaSuccess) {
        k_world_rays<<<blocks_for(rays, 256), 256, 0, s>>>(M.world, d_ins, d_angles, n, na, xyt);
        e = cudaGetLastError();
    }
    int rc = RLC_OK;
    if (e == cudaSuccess) rc = rlc_learned_predict(L, xyt, (int)rays, pred, stream);
    if (e == cudaSuccess && !rc) {
        k_resolve<<<blocks_for(rays, kResolveRays), kResolveThreads, 0, s>>>(M.map, M.mr, xyt, pred, (int)rays, M.world.s,
                                                                             d_outs, d_accepted, cnt);
        e = cudaGetLastError();
    }
    unsigned words[2] = {};
    if (e == cudaSuccess && !rc) e = M.take(words, s);
    if (rc) return rc;
    if (e != cudaSuccess) return lfail(RLC_ERR_CUDA, "learned ranges", e);
    if (words[0]) return lfail(RLC_ERR_CUDA, kTimedOut);   // predictions are missing: those of an older call were checked
    if (n_recast) *n_recast = (int)words[1];
    return RLC_OK;
}

// Test hook: C[M x N] (fp32, row-major) = A . B^T on the tensor cores, with A
// [M x K] (or K x M when a_t) and B [N x K] (or K x N when b_t), bf16, device.
int rlc_tc_gemm(const void* d_a, const void* d_b, float* d_c, int M, int N, int K, int a_t, int b_t, void* stream) {
    if (!d_a || !d_b || !d_c) return lfail(RLC_ERR_ARG, "null pointer");
    if (M <= 0 || N <= 0 || K <= 0 || M % kBM || N % kBN || K % tc::kKChunk)
        return lfail(RLC_ERR_ARG, "M must be a multiple of 128, N of 256, K of 64");
    unsigned* err = nullptr;
    const cudaStream_t s = (cudaStream_t)stream;
    LTRY(cudaMalloc(&err, sizeof(unsigned)), "gemm");
    cudaError_t e = cudaMemset(err, 0, sizeof(unsigned));
    bf16* copy[2] = {};   // of transposed operands that do not lie on the tile loads' 16 bytes
    auto aligned = [&](const void* p, size_t elems, int which) -> const bf16* {
        if (e != cudaSuccess || !((uintptr_t)p & 15)) return (const bf16*)p;
        e = cudaMalloc(&copy[which], elems * sizeof(bf16));
        if (e == cudaSuccess) e = cudaMemcpyAsync(copy[which], p, elems * sizeof(bf16), cudaMemcpyDeviceToDevice, s);
        return copy[which];
    };
    GemmArgs g{};
    g.A = a_t ? aligned(d_a, (size_t)M * K, 0) : (const bf16*)d_a; g.lda = a_t ? M : K; g.a_t = a_t != 0;   // [M x K], or [K x M]
    g.B = b_t ? aligned(d_b, (size_t)N * K, 1) : (const bf16*)d_b; g.ldb = b_t ? N : K; g.b_t = b_t != 0;
    g.M = M; g.N = N; g.K = K;
    g.ldc = N; g.C = d_c; g.err = err;
    if (e == cudaSuccess) e = gemm(g, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    unsigned h = 0;
    if (e == cudaSuccess) e = cudaMemcpy(&h, err, sizeof(unsigned), cudaMemcpyDeviceToHost);
    cudaFree(err);
    cudaFree(copy[0]);
    cudaFree(copy[1]);
    if (e != cudaSuccess) return lfail(RLC_ERR_CUDA, "tensor-core gemm", e);
    if (h) return lfail(RLC_ERR_CUDA, kTimedOut);
    return RLC_OK;
}

}  // extern "C"
