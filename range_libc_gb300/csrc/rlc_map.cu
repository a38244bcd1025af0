// Map preprocessing on the device: occupancy bit tiles, the exact Euclidean
// distance transform, the CDDT edge map and the tiled DT copy.
//
// Distance transform: the reference builds it on the CPU with the
// Felzenszwalb-Huttenlocher lower envelope (vendor/distance_transform.h:984-1030,
// called from RangeLib.h:345-373).  k_edt_pass_y/x run the same published
// algorithm, one thread per grid line, with the same float/double operation
// sequence so that every DT value is bit-identical: the intermediate sums
// f[q] + q*q are float (they round above 2^24, which matters on large
// maps), breakpoints are double, and the per-line output is a float.
// Pass 1 runs along y for every x, pass 2 along x for every y.  Maps with
// both sides <= 16384 take k_edt_cols/k_edt_rows instead: the same values from
// a search per cell (the argument is given above those kernels).
#include "rangelibc.h"
#include "rlc_internal.cuh"

#include <cfloat>
#include <cstdio>
#include <mutex>

namespace rlc {
namespace {

constexpr double kDblMax = 1.7976931348623157e308;

// bit j set where byte j of v is not 0
__device__ __forceinline__ unsigned nonzero_bytes(uint64_t v) {
    const uint64_t low = 0x7f7f7f7f7f7f7f7full;
    const uint64_t top = (((v & low) + low) | v) & ~low;                 // 0x80 in every such byte
    return (unsigned)(((top >> 7) * 0x0102040810204080ull) >> 56);
}

// Occupancy bytes to bit tiles, one thread per tile.  ROWS: the grid as image rows, occ[y * W + x]
// (numpy's [row, col]); otherwise occ[x * H + y].  A tile's eight lines of eight bytes are read as
// 8-byte words where the lines are aligned to them, and consecutive lanes read consecutive words:
// the grid may be host memory read in place over NVLink-C2C, so the transposition that image rows
// need costs nothing here (4.9 ms in numpy for 2048^2, 29 us for this kernel).
template <bool ROWS>
__global__ void __launch_bounds__(256) k_pack_bits(const uint8_t* __restrict__ occ, int W, int H, int TY,
                                                   uint64_t* __restrict__ bits) {
    const int TX = (W + 7) >> 3;
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= (long long)TX * TY) return;
    const int tx = ROWS ? (int)(t % TX) : (int)(t / TY), ty = ROWS ? (int)(t / TX) : (int)(t % TY);
    const int inner = ROWS ? W : H, outer = ROWS ? H : W;             // contiguous axis, line count
    const int i0 = (ROWS ? tx : ty) << 3, o0 = (ROWS ? ty : tx) << 3;
    const bool wide = i0 + 8 <= inner && inner % 8 == 0 && (reinterpret_cast<uintptr_t>(occ) & 7) == 0;
    uint64_t w = 0;
#pragma unroll
    for (int o = 0; o < 8; ++o) {
        if (o0 + o >= outer) break;
        const uint8_t* line = occ + (size_t)(o0 + o) * inner + i0;
        unsigned m = 0;
        if (wide) {
            m = nonzero_bytes(*reinterpret_cast<const uint64_t*>(line));
        } else {
            for (int i = 0; i < 8; ++i)
                if (i0 + i < inner && line[i]) m |= 1u << i;
        }
        if (ROWS) {   // line o is row y & 7 = o: its bits i are x & 7, at bit (i << 3) | o
            for (int i = 0; i < 8; ++i) w |= (uint64_t)((m >> i) & 1u) << ((i << 3) | o);
        } else {
            w |= (uint64_t)m << (o << 3);
        }
    }
    bits[(size_t)tx * TY + ty] = w;
}

// the tiles into host memory that the GPU writes in place: 512 KB for 2048^2, where a copy by the runtime into
// pageable memory took map creation 10 us longer
__global__ void __launch_bounds__(256) k_copy_bits(const uint64_t* __restrict__ bits, size_t words, uint64_t* __restrict__ out) {
    for (size_t i = (size_t)blockIdx.x * 256 + threadIdx.x; i < words; i += (size_t)gridDim.x * 256) out[i] = bits[i];
}

__device__ __forceinline__ bool occ_bit(const uint64_t* __restrict__ bits, int TY, int x, int y) {
    uint64_t w = bits[(size_t)(x >> 3) * TY + (y >> 3)];
    return (w >> (((x & 7) << 3) | (y & 7))) & 1ull;
}

// One F-H line.  f(q) is the input sample q, out(q, value) stores the
// output; v/z are this line's scratch arrays with a stride of `ld` elements
// between consecutive k (lines interleave so that neighbouring threads touch
// neighbouring words).
template <class In, class Out>
__device__ void fh_line(const In& f, const Out& out, unsigned n, uint32_t* v, double* z, size_t ld) {
    if (n == 0) return;
    if (n == 1) { out(0, f(0)); return; }
    unsigned k = 0;
    v[0] = 0;
    z[0] = -kDblMax;
    z[ld] = kDblMax;
    for (unsigned q = 1; q < n; ++q) {
        double s;
        float fq = __fadd_rn(f(q), __ull2float_rn((unsigned long long)q * q));
        double dq2 = __ull2double_rn(2ull * q);
        ++k;
        do {
            --k;
            unsigned vk = v[(size_t)k * ld];
            float fv = __fadd_rn(f(vk), __ull2float_rn((unsigned long long)vk * vk));
            s = __ddiv_rn(__dsub_rn((double)fq, (double)fv), __dsub_rn(dq2, __ull2double_rn(2ull * vk)));
        } while (s <= z[(size_t)k * ld]);
        ++k;
        v[(size_t)k * ld] = q;
        z[(size_t)k * ld] = s;
        z[(size_t)(k + 1) * ld] = kDblMax;
    }
    k = 0;
    for (unsigned q = 0; q < n; ++q) {
        while (z[(size_t)(k + 1) * ld] < __uint2double_rn(q)) ++k;
        unsigned vk = v[(size_t)k * ld];
        float dq = __fsub_rn(__uint2float_rn(q), __uint2float_rn(vk));
        out(q, __fadd_rn(f(vk), __fmul_rn(dq, dq)));
    }
}

struct OccInput {           // pass 1 input along y for a fixed x
    const uint64_t* bits; int TY; int x;
    __device__ float operator()(unsigned q) const { return occ_bit(bits, TY, x, (int)q) ? 0.0f : FLT_MAX; }
};
struct ColOutput {          // pass 1 output g[x * H + q]
    float* g; size_t base;
    __device__ void operator()(unsigned q, float val) const { g[base + q] = val; }
};
struct RowInput {           // pass 2 input along x for a fixed y: g[q * H + y]
    const float* g; int H; int y;
    __device__ float operator()(unsigned q) const { return g[(size_t)q * H + y]; }
};
struct RowSqrtOutput {      // pass 2 output: sqrt, element_wiseSquareRoot
    float* dt; int H; int y;
    __device__ void operator()(unsigned q, float val) const { dt[(size_t)q * H + y] = __fsqrt_rn(val); }
};

__global__ void k_edt_pass_y(const uint64_t* __restrict__ bits, int W, int H, int TY, float* g,
                             uint32_t* v, double* z) {
    int x = blockIdx.x * blockDim.x + threadIdx.x;
    if (x >= W) return;
    fh_line(OccInput{bits, TY, x}, ColOutput{g, (size_t)x * H}, (unsigned)H, v + x, z + x, (size_t)W);
}

__global__ void k_edt_pass_x(const float* g, int W, int H, float* dt, uint32_t* v, double* z) {
    int y = blockIdx.x * blockDim.x + threadIdx.x;
    if (y >= H) return;
    fh_line(RowInput{g, H, y}, RowSqrtOutput{dt, H, y}, (unsigned)W, v + y, z + y, (size_t)H);
}

// ---- maps with both sides <= 16384 -------------------------------------------------------------
//
// For such maps a cheaper computation of the F-H steps above gives the same results bit for bit.
// Every finite key K(q) = f(q) + q*q (a float sum, as in the reference) is an integer below 2^29,
// and every breakpoint is a quotient a / b of integers with |a| < 2^29 and 2 <= b <= 2 (n - 1) <
// 2^15, computed in double exactly up to the final rounding.  Rounding moves a / b by at most
// 2^-53 |a| / b, while two different quotients a / b and c / d differ by at least 1 / (b d);
// since |a| d + |c| b < 2^45 < 2^53, rounding never reverses or merges two different quotients,
// and equal quotients round alike.  A comparison of rounded breakpoints (s <= z[k],
// z[k + 1] < q) therefore has the outcome of the exact comparison of the quotients.
//  * edt_col_exact and fh_line_exact are the reference's steps with those comparisons decided in
//    integers, one line after the other; comparisons with a FLT_MAX key run in double as in the
//    reference.  No kernel runs them: they are this rule as code, checked against the reference's
//    transform on the host (tests/cpp/edt_exact_check.cu).  The searches that the kernels run are
//    checked against that transform by themselves (edt_search_check.cu, edt_search_maps.cu).
//  * So the envelope is the exact lower envelope of the lines K(p) - 2 p q, and at an integer q it
//    takes the smallest p among those with the least K(p) - 2 p q: `s <= z[k]` drops a vertex that
//    is nowhere strictly least, `z[k + 1] < q` stays with the left vertex where two tie.  A
//    FLT_MAX vertex is never taken while a finite one exists (its breakpoints lie beyond
//    +-FLT_MAX / 2^15), and a line without a finite input gives FLT_MAX.
//  * K(p) - 2 p q + q*q = f(p) + (p - q)^2 + e(p), where e(p) is what rounding added to the key: 0
//    while keys stay below 2^24, at most 1 below 2^25 (sides <= 4096: q*q is exact), at most
//    8 + 16 below 2^29.  Since f >= 0, no vertex further from q than the square root of (the least
//    value found so far + the bound of e) can be least: each cell is found by searching outward
//    from it, all cells in parallel (edt_col_search, edt_row_search).
constexpr int kEdtExactSide = 4096;           // q*q is exact
constexpr int kEdtIntSide = 16384;            // integer comparisons
constexpr float kEdtExactKey = 536870912.0f;  // 2^29: finite keys are below it

__host__ __device__ __forceinline__ float edt_fadd(float a, float b) {
#ifdef __CUDA_ARCH__
    return __fadd_rn(a, b);
#else
    return a + b;
#endif
}
__host__ __device__ __forceinline__ float edt_fsub(float a, float b) {
#ifdef __CUDA_ARCH__
    return __fsub_rn(a, b);
#else
    return a - b;
#endif
}
__host__ __device__ __forceinline__ float edt_fmul(float a, float b) {
#ifdef __CUDA_ARCH__
    return __fmul_rn(a, b);
#else
    return a * b;
#endif
}
// f(v) + v*v in float, as the reference sums it (v*v < 2^32)
__host__ __device__ __forceinline__ float edt_key(float fv, unsigned v) { return edt_fadd(fv, (float)(v * v)); }
// the reference's breakpoint ((double)kb - (double)ka) / ((double)(2 b) - (double)(2 a))
__host__ __device__ __forceinline__ double edt_isect(float ka, unsigned a, float kb, unsigned b) {
#ifdef __CUDA_ARCH__
    return __ddiv_rn(__dsub_rn((double)kb, (double)ka),
                     __dsub_rn(__ull2double_rn(2ull * b), __ull2double_rn(2ull * a)));
#else
    return ((double)kb - (double)ka) / ((double)(2ull * b) - (double)(2ull * a));
#endif
}
__host__ __device__ __forceinline__ int edt_lsb(unsigned b) {   // b != 0
#ifdef __CUDA_ARCH__
    return __ffs(b) - 1;
#else
    return __builtin_ctz(b);
#endif
}
__host__ __device__ __forceinline__ int edt_msb(unsigned b) {   // b != 0
#ifdef __CUDA_ARCH__
    return 31 - __clz(b);
#else
    return 31 - __builtin_clz(b);
#endif
}

// Pass 1 of one column (H <= 4096).  col[c] is the bit tile of rows 8c..8c+7, the column's byte at
// bit offset sh; nx holds TY + 1 entries of scratch; out[q] receives the squared distance.
__host__ __device__ inline void edt_col_exact(const uint64_t* col, int sh, int H, int TY, uint16_t* nx,
                                              float* out) {
    constexpr unsigned kNone = 0xFFFFu;
    unsigned nxt = kNone;   // first occupied row at or after 8c
    nx[TY] = (uint16_t)kNone;
    for (int c = TY - 1; c >= 0; --c) {
        const unsigned b = (unsigned)(col[c] >> sh) & 0xFFu;
        if (b) nxt = ((unsigned)c << 3) + (unsigned)edt_lsb(b);
        nx[c] = (uint16_t)nxt;
    }
    int prev = -1;          // last occupied row before 8c
    for (int c = 0; c < TY; ++c) {
        const unsigned b = (unsigned)(col[c] >> sh) & 0xFFu;
        const unsigned beyond = nx[c + 1];
        const int base = c << 3, m = H - base < 8 ? H - base : 8;
        for (int j = 0; j < m; ++j) {
            const int q = base + j;
            const unsigned lo = b & ((2u << j) - 1u), hi = b >> j;
            const int p = lo ? base + edt_msb(lo) : prev;
            const unsigned nq = hi ? (unsigned)(q + edt_lsb(hi)) : beyond;
            int d = 0x7FFFFFFF;
            if (p >= 0) d = q - p;
            if (nq != kNone && (int)nq - q < d) d = (int)nq - q;
            out[q] = d == 0x7FFFFFFF ? FLT_MAX : (float)(d * d);
        }
        if (b) prev = base + edt_msb(b);
    }
}

// One line (both sides <= 16384): the reference's F-H steps with the comparisons decided exactly.
// The stack's entry k is (sv[k * ld], sf[k * ld]) -- vertex and its input value -- with room for
// n entries; the top two entries are also kept in registers.
#pragma nv_exec_check_disable
template <class In, class Out>
__host__ __device__ void fh_line_exact(const In& f, const Out& out, unsigned n, uint16_t* sv, float* sf,
                                       size_t ld) {
    if (n == 0) return;
    if (n == 1) { out(0, f(0)); return; }
    unsigned top = 0, vt = 0, vs = 0;   // (vt, kt) entry top, (vs, ks) entry top - 1
    const float f0 = f(0);
    sv[0] = 0;
    sf[0] = f0;
    float kt = edt_key(f0, 0), ks = 0.0f, fnext = f(1);
    for (unsigned q = 1; q < n; ++q) {
        const float fq = fnext;
        if (q + 1 < n) fnext = f(q + 1);
        const float kq = edt_key(fq, q);
        while (top > 0) {   // z[0] = -DBL_MAX: the bottom vertex is never popped
            bool pop;
            if (kq < kEdtExactKey && kt < kEdtExactKey && ks < kEdtExactKey)
                pop = (long long)((int)kq - (int)kt) * (int)(vt - vs) <=
                      (long long)((int)kt - (int)ks) * (int)(q - vt);
            else
                pop = edt_isect(kt, vt, kq, q) <= edt_isect(ks, vs, kt, vt);
            if (!pop) break;
            --top;
            vt = vs;
            kt = ks;
            if (top > 0) {
                vs = sv[(size_t)(top - 1) * ld];
                ks = edt_key(sf[(size_t)(top - 1) * ld], vs);
            }
        }
        ++top;
        sv[(size_t)top * ld] = (uint16_t)q;
        sf[(size_t)top * ld] = fq;
        vs = vt;
        ks = kt;
        vt = q;
        kt = kq;
    }
    unsigned k = 0, vk = sv[0], vn = 0;
    float fk = sf[0], kk = edt_key(fk, vk), fn = 0.0f;
    if (top > 0) {
        vn = sv[ld];
        fn = sf[ld];
    }
    for (unsigned q = 0; q < n; ++q) {
        while (k < top) {   // z[top + 1] = DBL_MAX; (vn, fn) is entry k + 1
            const float kn = edt_key(fn, vn);
            bool adv;
            if (kk < kEdtExactKey && kn < kEdtExactKey)
                adv = (long long)((int)kn - (int)kk) < (long long)q * (long long)(2u * (vn - vk));
            else
                adv = edt_isect(kk, vk, kn, vn) < (double)q;
            if (!adv) break;
            ++k;
            vk = vn;
            fk = fn;
            kk = kn;
            if (k < top) {
                vn = sv[(size_t)(k + 1) * ld];
                fn = sf[(size_t)(k + 1) * ld];
            }
        }
        const float dq = edt_fsub((float)q, (float)vk);
        out(q, edt_fadd(fk, edt_fmul(dq, dq)));
    }
}

// ---- the searches
constexpr unsigned kEdtNone = 0xFFFFu;   // "no occupied cell in the column"
constexpr int kEdtNear = 8;              // distances searched one by one before whole blocks
constexpr int kEdtBlock = 8;             // cells of a row whose least pass-1 distance is kept together,
constexpr int kEdtFar = 64;              // and whose least blocks' distance is, for the search beyond kEdtFar

// f of a pass-1 distance d: the float square (pass 1 stores 0 + (q - v)^2), FLT_MAX for none
__host__ __device__ __forceinline__ float edt_f(unsigned d) {
    return d == kEdtNone ? FLT_MAX : edt_fmul((float)d, (float)d);
}

// Pass 1 at row q: the distance to the vertex F-H takes.  prev / next: the last occupied row <= q
// (-1: none) and the first >= q (kEdtNone: none).  Up to 4096 rows that is the nearest of them;
// above, q*q rounds (e <= 8 either way), so that a vertex up to sqrt(d*d + 16) away can win.
template <class Occ>
__host__ __device__ __forceinline__ unsigned edt_col_search(int prev, unsigned next, int q, int H, const Occ& occ) {
    int d = 0x7FFFFFFF;
    if (prev >= 0) d = q - prev;
    if (next != kEdtNone && (int)next - q < d) d = (int)next - q;
    if (d == 0x7FFFFFFF) return kEdtNone;
    if (H <= kEdtExactSide) return (unsigned)d;
    const int limit = d * d + 16;
    int best = 0x7FFFFFFF, at = 0;
    for (int e = d; e * e <= limit; ++e)
        for (int side = 0; side < 2; ++side) {
            const int p = side ? q + e : q - e;
            if (p < 0 || p >= H || !occ(p)) continue;
            const int cost = (int)(float)(p * p) - 2 * p * q;
            if (cost < best || (cost == best && p < at)) {
                best = cost;
                at = p;
            }
        }
    return (unsigned)(at < q ? q - at : at - q);
}

// The blocks beyond kEdtNear of q in growing distance, until near(gap) says that columns `gap` or more away
// cannot win; columns(first, end) looks into a block for which worth(gap, its least distance) holds.
template <class Near, class Worth, class Columns, class GMin, class GFar>
__host__ __device__ __forceinline__ void edt_blocks(const Near& near, const Worth& worth, const Columns& columns,
                                                    const GMin& gmin, const GFar& gfar, int W, int q) {
    const int nb = (W + kEdtBlock - 1) / kEdtBlock, nf = (W + kEdtFar - 1) / kEdtFar, ratio = kEdtFar / kEdtBlock;
    auto block = [&](int b) {
        const int gap = b * kEdtBlock > q ? b * kEdtBlock - q : q - (b * kEdtBlock + kEdtBlock - 1);
        if (!near(gap)) return false;
        const unsigned m = gmin(b);
        if (m != kEdtNone && worth(gap, m)) columns(b * kEdtBlock, b * kEdtBlock + kEdtBlock < W ? b * kEdtBlock + kEdtBlock : W);
        return true;
    };
    bool open = true;
    for (int k = 1, own = q / kEdtBlock; k <= ratio && open; ++k) {
        open = own - k >= 0 && block(own - k);
        if (own + k < nb && block(own + k)) open = true;
    }
    for (int k = 1, own = q / kEdtFar; open; ++k) {
        open = false;
        for (int side = 0; side < 2; ++side) {
            const int f = side ? own + k : own - k;
            if (f < 0 || f >= nf) continue;
            const int gap = side ? f * kEdtFar - q : q - (f * kEdtFar + kEdtFar - 1);
            if (!near(gap)) continue;
            open = true;
            const unsigned m = gfar(f);
            if (m == kEdtNone || !worth(gap, m)) continue;
            for (int b = f * ratio; b < (f + 1) * ratio && b < nb; ++b) (void)block(b);
        }
    }
}

// Pass 2 at column q of a row of W pass-1 distances g(p): the value whose square root is the
// distance transform.  gmin(b): the least distance of columns [8 b, 8 b + 8), gfar(b) of [64 b, 64 b + 64).
// Distances up to kEdtNear are searched one by one, then blocks of 8 columns up to 64, then of 64, each
// looked into only where its least distance could win: a cell 50 px from the walls asks 14 blocks and not
// 100 columns, and an empty map costs W / 64 reads per cell.  Map and marcher set up, us, one by one to 32
// and blocks of 32 / this: corridor 2048^2 382 / 343, rectangles and disks 368 / 340, 8192^2 5819 / 4570, a
// single obstacle 578 / 468 (with blocks of 8 alone 338, 342, 4550, 941).
//
// Keys below 2^24: the value is the least f(p) + (p - q)^2, and which p gives it does not matter.
// So the near search runs in groups of four distances with one exit test, and a position past the
// row's end reads its last cell instead (which at that distance is never less than it is itself).
template <class G, class GMin, class GFar>
__host__ __device__ __forceinline__ float edt_row_search_exact(const G& g, const GMin& gmin, const GFar& gfar, int W, int q) {
    // 65535^2 + e^2 < 2^32 for e <= 256 stands for "none"; every true value is below 2^24
    unsigned best = g(q) * g(q);
    int e = 1;
    for (; e <= kEdtNear && (unsigned)(e * e) < best; e += 4) {
        unsigned d[8];
#ifdef __CUDA_ARCH__
#pragma unroll
#endif
        for (int u = 0; u < 4; ++u) {
            d[2 * u] = g(q - e - u > 0 ? q - e - u : 0);
            d[2 * u + 1] = g(q + e + u < W ? q + e + u : W - 1);
        }
#ifdef __CUDA_ARCH__
#pragma unroll
#endif
        for (int u = 0; u < 4; ++u) {
            const unsigned e2 = (unsigned)((e + u) * (e + u));
            const unsigned l = d[2 * u] * d[2 * u] + e2, r = d[2 * u + 1] * d[2 * u + 1] + e2;
            const unsigned m = l < r ? l : r;
            best = m < best ? m : best;
        }
    }
    if (e > kEdtNear && (unsigned)(e * e) < best)
        edt_blocks([&](int gap) { return (unsigned)(gap * gap) < best; },
                   [&](int gap, unsigned m) { return (unsigned)(gap * gap) + m * m < best; },
                   [&](int p, int end) {
                       for (; p < end; ++p) {
                           const unsigned d = g(p), c = d * d + (unsigned)((p - q) * (p - q));
                           best = d != kEdtNone && c < best ? c : best;
                       }
                   },
                   gmin, gfar, W, q);
    return best < (1u << 24) ? (float)best : FLT_MAX;
}

// Keys that round: they are formed as the reference rounds them, `slack` bounds e, and the smallest
// p of the least keys is the one taken.
template <class G, class GMin, class GFar>
__host__ __device__ __forceinline__ float edt_row_search_rounded(const G& g, const GMin& gmin, const GFar& gfar, int W, int q,
                                                                  int slack) {
    int best = 0x7FFFFFFF, at = q;   // best: K(p) - 2 p q + q q
    unsigned d_at = kEdtNone;
    auto take = [&](int p) {
        const unsigned d = g(p);
        if (d == kEdtNone) return;
        const int cost = (int)edt_key(edt_f(d), (unsigned)p) - 2 * p * q + q * q;
        if (cost < best || (cost == best && p < at)) {
            best = cost;
            at = p;
            d_at = d;
        }
    };
    take(q);
    int e = 1;
    for (; e <= kEdtNear && e * e - slack <= best; ++e) {
        if (q - e >= 0) take(q - e);
        if (q + e < W) take(q + e);
    }
    if (e > kEdtNear && e * e - slack <= best)
        edt_blocks([&](int gap) { return gap * gap - slack <= best; },
                   [&](int gap, unsigned m) { return gap * gap - slack <= best - (int)edt_f(m); },
                   [&](int p, int end) {
                       for (; p < end; ++p) take(p);
                   },
                   gmin, gfar, W, q);
    if (d_at == kEdtNone) return FLT_MAX;
    const float dq = edt_fsub((float)q, (float)at);
    return edt_fadd(edt_f(d_at), edt_fmul(dq, dq));
}

template <bool EXACT, class G, class GMin, class GFar>
__host__ __device__ __forceinline__ float edt_row_search(const G& g, const GMin& gmin, const GFar& gfar, int W, int q, int slack) {
    return EXACT ? edt_row_search_exact(g, gmin, gfar, W, q) : edt_row_search_rounded(g, gmin, gfar, W, q, slack);
}

// Pass 1, a few blocks per 8 columns (a row of bit tiles), each answering a share of the rows.  Bound by its 2 bytes per cell written.  A
// warp per column finds, for every tile, the last occupied row before it and the first one at or
// after it (a ballot per 32 tiles); every thread then answers its rows from the tile's byte and
// those two.  2048^2: 121 us with one thread per column -> 17 us.
__global__ void __launch_bounds__(256) k_edt_cols(const uint64_t* __restrict__ bits, int W, int H, int TY,
                                                  uint16_t* __restrict__ g) {
    extern __shared__ uint16_t s_near[];   // per column: before[TY], from[TY]
    const int tx = blockIdx.x, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint64_t* col = bits + (size_t)tx * TY;
    const unsigned full = 0xffffffffu;
    {
        uint16_t* before = s_near + (size_t)warp * 2 * TY;
        uint16_t* from = before + TY;
        const int chunks = (TY + 31) >> 5, sh = warp << 3;
        unsigned carry = kEdtNone;
        for (int k = 0; k < chunks; ++k) {
            const int c = (k << 5) + lane;
            const unsigned b = c < TY ? (unsigned)(col[c] >> sh) & 0xFFu : 0u;
            const unsigned row = b ? ((unsigned)c << 3) + (unsigned)edt_msb(b) : 0u;
            const unsigned mask = __ballot_sync(full, b != 0), below = mask & ((1u << lane) - 1u);
            const unsigned v = __shfl_sync(full, row, below ? 31 - __clz(below) : 0);
            if (c < TY) before[c] = (uint16_t)(below ? v : carry);
            const unsigned lastv = __shfl_sync(full, row, mask ? 31 - __clz(mask) : 0);
            if (mask) carry = lastv;
        }
        carry = kEdtNone;
        for (int k = chunks - 1; k >= 0; --k) {
            const int c = (k << 5) + lane;
            const unsigned b = c < TY ? (unsigned)(col[c] >> sh) & 0xFFu : 0u;
            const unsigned row = b ? ((unsigned)c << 3) + (unsigned)edt_lsb(b) : 0u;
            const unsigned mask = __ballot_sync(full, b != 0), at = mask & ~((1u << lane) - 1u);
            const unsigned v = __shfl_sync(full, row, at ? __ffs(at) - 1 : 0);
            if (c < TY) from[c] = (uint16_t)(at ? v : carry);
            const unsigned firstv = __shfl_sync(full, row, mask ? __ffs(mask) - 1 : 0);
            if (mask) carry = firstv;
        }
    }
    __syncthreads();
    for (int j = 0; j < 8; ++j) {
        const int x = (tx << 3) + j;
        if (x >= W) break;
        const uint16_t* before = s_near + (size_t)j * 2 * TY;
        const uint16_t* from = before + TY;
        const auto occ = [&](int p) { return (col[p >> 3] >> ((j << 3) | (p & 7))) & 1ull; };
        for (int q = blockIdx.y * blockDim.x + threadIdx.x; q < H; q += gridDim.y * blockDim.x) {
            const int c = q >> 3, in = q & 7;
            const unsigned b = (unsigned)(col[c] >> (j << 3)) & 0xFFu;
            const unsigned lo = b & ((2u << in) - 1u), hi = b >> in;
            int prev = lo ? (c << 3) + edt_msb(lo) : (before[c] == kEdtNone ? -1 : (int)before[c]);
            unsigned next = hi ? (unsigned)(q + edt_lsb(hi)) : (c + 1 < TY ? from[c + 1] : kEdtNone);
            g[(size_t)x * H + q] = (uint16_t)edt_col_search(prev, next, q, H, occ);
        }
    }
}

// the least pass-1 distance of every block of kEdtBlock columns and of every kEdtFar, per row:
// gmin[b * H + y], gfar[b * H + y]
__global__ void __launch_bounds__(256) k_edt_block_min(const uint16_t* __restrict__ g, int W, int H,
                                                       uint16_t* __restrict__ gmin, uint16_t* __restrict__ gfar) {
    const int y = blockIdx.x * blockDim.x + threadIdx.x, f = blockIdx.y;
    if (y >= H) return;
    unsigned least = kEdtNone;
    for (int b = f * (kEdtFar / kEdtBlock); b < (f + 1) * (kEdtFar / kEdtBlock) && b * kEdtBlock < W; ++b) {
        unsigned m = kEdtNone;
#pragma unroll
        for (int j = 0; j < kEdtBlock; ++j) m = min(m, (unsigned)__ldg(g + (size_t)min(b * kEdtBlock + j, W - 1) * H + y));
        gmin[(size_t)b * H + y] = (uint16_t)m;
        least = min(least, m);
    }
    gfar[(size_t)f * H + y] = (uint16_t)least;
}

// Every form of the distance transform at cell (x, y), value dt; padding cells of the tiles too.
//  * tiled: the float in 8x8 tiles (0 in the padding);
//  * u16: d^2 in 8x8 tiles, 4x4 cells per 32-byte sector, u8: d^2 in 8x8 tiles of 64 bytes; all
//    ones = "read the float" (and in the padding).  dt = sqrtf(D) of an integer D, and for D <
//    2^16 the float product dt * dt is within 0.02 of it;
//  * step: the march step max(dt * 0.999, 1) of RangeLib.h:957, NaN on occupied cells, in a grid
//    with one more row and column of +inf (what a march off the grid reads).
__device__ __forceinline__ void store_layouts(const DtOut& o, int W, int H, int TY, int x, int y, float dt) {
    const bool in = x < W && y < H;
    const size_t tile = ((size_t)(x >> 3) * TY + (y >> 3)) << 6;
    const float d2 = rintf(__fmul_rn(dt, dt));
    if (in) {
        const size_t i = (size_t)x * H + y;
        o.dt[i] = dt;
        if (o.step) {
            const float v = __fmul_rn(dt, 0.999f), inf = __int_as_float(0x7f800000);
            float* row = o.step + (size_t)x * (H + 1);
            row[y] = dt <= 0.0f ? __int_as_float(0x7fc00000) : (v < 1.0f ? 1.0f : v);
            if (y == H - 1) row[H] = inf;
            if (x == W - 1) row[H + 1 + y] = inf;
            if (x == W - 1 && y == H - 1) row[H + 1 + H] = inf;
        }
    }
    o.tiled[tile + ((x & 7) << 3) + (y & 7)] = in ? dt : 0.0f;
    o.u16[tile + ((((x >> 2) & 1) << 1 | ((y >> 2) & 1)) << 4) + (((x & 3) << 2) | (y & 3))] =
        in && d2 < 65535.0f ? (uint16_t)d2 : (uint16_t)0xFFFF;
    o.u8[tile + ((x & 7) << 3) + (y & 7)] = in && d2 <= 254.0f ? (uint8_t)d2 : (uint8_t)0xFF;
}

// Pass 2, one thread per cell, 32 consecutive y per warp (the searched distances of a warp are
// whole 64-byte pieces) x 8 x per block (which share them in the L1).  Bound by the search's
// instructions: up to 17 reads of columns per cell, then one for each block of 8 up to 64 columns away and
// of 64 beyond, and the columns of those that could win.  ALL: writes every layout, straight from
// the search (60 MB at 2048^2; four more kernels read the linear one back before).
// 2048^2 with the layouts: 1553 + 117 us with one thread per row, 121 with blocks of 32 columns, now 88.
template <bool EXACT, bool ALL>
__global__ void __launch_bounds__(256) k_edt_rows(const uint16_t* __restrict__ g, const uint16_t* __restrict__ gmin,
                                                  const uint16_t* __restrict__ gfar,
                                                  int W, int H, int TY, int slack, DtOut o) {
    const int y = blockIdx.x * 32 + threadIdx.x, x = blockIdx.y * 8 + threadIdx.y;
    float dt = 0.0f;
    if (x < W && y < H)
        dt = __fsqrt_rn(edt_row_search<EXACT>([&](int p) { return (unsigned)__ldg(g + (size_t)p * H + y); },
                                              [&](int b) { return (unsigned)__ldg(gmin + (size_t)b * H + y); },
                                              [&](int b) { return (unsigned)__ldg(gfar + (size_t)b * H + y); }, W, x,
                                              slack));
    if (ALL) {
        if ((y >> 3) < TY) store_layouts(o, W, H, TY, x, y, dt);
    } else if (x < W && y < H) {
        o.dt[(size_t)x * H + y] = dt;
    }
}

// the layouts of a linear distance transform (maps with a side above 16384)
__global__ void __launch_bounds__(256) k_dt_layouts(const float* __restrict__ lin, int W, int H, int TY, DtOut o) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const int TX = (W + 7) >> 3;
    if (i >= (long long)TX * TY * 64) return;
    const long long tile = i >> 6;
    const int within = (int)(i & 63), tx = (int)(tile / TY), ty = (int)(tile - (long long)tx * TY);
    const int x = (tx << 3) + (within >> 3), y = (ty << 3) + (within & 7);
    store_layouts(o, W, H, TY, x, y, x < W && y < H ? lin[(size_t)x * H + y] : 0.0f);
}

// ---- equal-step runs
// Which neighbouring cells have equal steps, one bit per cell and axis: bit y & 31 of eqy[x * HW +
// (y >> 5)] is step(x, y - 1) == step(x, y), bit x & 31 of eqx[(x >> 5) * H + y] is step(x - 1, y)
// == step(x, y).  A warp reads a 32 x 32 patch once, 32 independent coalesced rows.
__global__ void __launch_bounds__(256) k_step_eq(const float* __restrict__ step, int W, int H, int HW,
                                                 uint32_t* __restrict__ eqx, uint32_t* __restrict__ eqy,
                                                 unsigned long long* __restrict__ share) {
    const long long w = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (w == 0 && threadIdx.x == 0) *share = 0ull;
    const int lane = threadIdx.x & 31, XW = (W + 31) >> 5;
    if (w >= (long long)XW * HW) return;
    const int xw = (int)(w / HW), yw = (int)(w - (long long)xw * HW), x0 = xw << 5, y = (yw << 5) + lane;
    const size_t pitch = (size_t)H + 1;   // of the step map
    const bool in = y < H;
    const float none = __int_as_float(0x7fc00000);   // equal to nothing
    // lane j: the cell before this patch's rows in column x0 + j
    const float edge = yw > 0 && x0 + lane < W ? __ldg(step + (x0 + lane) * pitch + (yw << 5) - 1) : none;
    float prev = in && x0 > 0 ? __ldg(step + (x0 - 1) * pitch + y) : none;
    uint32_t mx = 0, my = 0;
#pragma unroll
    for (int j0 = 0; j0 < 32; j0 += 8) {
        float v[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) v[j] = in && x0 + j0 + j < W ? __ldg(step + (x0 + j0 + j) * pitch + y) : none;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            float left = __shfl_up_sync(0xffffffffu, v[j], 1);
            const float before = __shfl_sync(0xffffffffu, edge, j0 + j);
            if (lane == 0) left = before;
            const uint32_t m = __ballot_sync(0xffffffffu, left == v[j]);
            if (lane == j0 + j) my = m;   // lane j keeps column x0 + j's word
            mx |= (uint32_t)(prev == v[j]) << (j0 + j);
            prev = v[j];
        }
    }
    if (x0 + lane < W) eqy[(size_t)(x0 + lane) * HW + yw] = my;
    if (in) eqx[(size_t)xw * H + y] = mx;
}

// consecutive set bits at position j and below (down) or at j and above (up) of a bit line whose
// word w is word(w), at most 255; up stops at the line's end (nw words)
template <class Word>
__device__ __forceinline__ unsigned bits_down(const Word& word, int j) {
    unsigned n = 0;
    for (int w = j >> 5, l = j & 31;; --w, l = 31) {
        const unsigned t = (unsigned)__clz((int)~(word(w) << (31 - l)));
        n += min(t, (unsigned)(l + 1));
        if (t < (unsigned)(l + 1) || w == 0 || n >= 255u) break;
    }
    return min(n, 255u);
}
template <class Word>
__device__ __forceinline__ unsigned bits_up(const Word& word, int j, int nw) {
    unsigned n = 0;
    for (int w = j >> 5, l = j & 31; w < nw; ++w, l = 0) {
        const unsigned z = ~(word(w) >> l), t = min(z ? (unsigned)__ffs((int)z) - 1u : 32u, 32u - (unsigned)l);
        n += t;
        if (t < 32u - (unsigned)l || n >= 255u) break;
    }
    return min(n, 255u);
}

// runs[x * H + y]: how many cells after (x, y) along +y, -y, +x and -x have its step (bits 0-7,
// 8-15, 16-23, 24-31; at most 255 each), counted in the bit lines: one or two words per direction
// where a thread per line walked the map before.  2048^2: 2106 us -> 51 us with k_step_eq.
// *share, zeroed before: over a sixteenth of the blocks, the free cells (upper half) and those of them with
// a run that a ray may skip (kLongRun; lower half).
constexpr uint32_t kLongRun = 12;

__global__ void __launch_bounds__(256) k_step_runs(const uint32_t* __restrict__ eqx, const uint32_t* __restrict__ eqy,
                                                   const float* __restrict__ step, int W, int H, int HW,
                                                   uint32_t* __restrict__ runs, unsigned long long* __restrict__ share) {
    const unsigned yb = ((unsigned)H + 31u) >> 5, bx = blockIdx.x / yb;   // 32 y x 8 x cells per block
    const int x = (int)(bx * 8 + threadIdx.y), y = (int)((blockIdx.x - bx * yb) * 32 + threadIdx.x);
    const bool in = x < W && y < H;
    uint32_t word = 0;
    if (in) {
        const auto wx = [&](int w) { return __ldg(eqx + (size_t)w * H + y); };
        const auto wy = [&](int w) { return __ldg(eqy + (size_t)x * HW + w); };
        word = bits_up(wy, y + 1, HW) | bits_down(wy, y) << 8 | bits_up(wx, x + 1, (W + 31) >> 5) << 16 |
               bits_down(wx, x) << 24;
        runs[(size_t)x * H + y] = word;
    }
    if ((blockIdx.x * 0x9E3779B1u) >> 28) return;
    const int free = __syncthreads_count(in && !isnan(__ldg(step + (size_t)x * (H + 1) + y)));
    const int lng = __syncthreads_count(in && __vcmpgeu4(word, kLongRun * 0x01010101u) != 0u);
    if (threadIdx.x == 0 && threadIdx.y == 0 && free) atomicAdd(share, ((unsigned long long)free << 32) + (unsigned)lng);
}

// RangeLib.h:293-312: an occupied cell with any in-grid free 8-neighbour.
__global__ void k_edge_map(const uint64_t* __restrict__ bits, int W, int H, int TY, uint8_t* __restrict__ edge) {
    long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= (long long)W * H) return;
    int x = (int)(i / H), y = (int)(i - (long long)x * H);
    uint8_t e = 0;
    if (occ_bit(bits, TY, x, y)) {
        for (int dx = -1; dx <= 1 && !e; ++dx)
            for (int dy = -1; dy <= 1; ++dy) {
                if (!dx && !dy) continue;
                int cx = x + dx, cy = y + dy;
                if (cx >= 0 && cy >= 0 && cx < W && cy < H && !occ_bit(bits, TY, cx, cy)) { e = 1; break; }
            }
    }
    edge[i] = e;
}

// ---- free distances (Bresenham's walk)
// Distance along y from cell (x, y) to the nearest occupied cell of its column, at most kFreeMost: the
// bytes of the column's tiles, outward.
__device__ __forceinline__ int free_y(const uint64_t* __restrict__ bits, int TY, int x, int y) {
    const uint64_t* col = bits + (size_t)(x >> 3) * TY;
    const int sh = (x & 7) << 3, c = y >> 3, in = y & 7;
    const unsigned b = (unsigned)(__ldg(col + c) >> sh) & 0xFFu;
    const unsigned lo = b & ((2u << in) - 1u), hi = b >> in;
    int d = kFreeMost;
    if (lo) d = min(d, in - edt_msb(lo));
    if (hi) d = min(d, edt_lsb(hi));
    for (int k = 1; 8 * k - 7 < d && (c - k >= 0 || c + k < TY); ++k) {
        const unsigned l = c - k >= 0 ? (unsigned)(__ldg(col + c - k) >> sh) & 0xFFu : 0u;
        const unsigned r = c + k < TY ? (unsigned)(__ldg(col + c + k) >> sh) & 0xFFu : 0u;
        if (l) d = min(d, 8 * k + in - edt_msb(l));
        if (r) d = min(d, 8 * k - in + edt_lsb(r));
    }
    return d;
}

// Chebyshev distance: the least over dx of max(|dx|, distance along y at x + dx); a (W + 1) x (H + 1) grid
// with 1 in its last row and column.  A block answers kFreeTile x 32 cells from the distances along y of
// their columns and of kFreeMost - 1 on either side, in shared memory, so that the map needs no scratch
// beside its result (two passes with one in memory before: a method on 2048^2 with walls made in 219 us, now
// 190; with blocks of 8 warps, each on its rows in turn, 220, and 86 instead of 49 on 512^2).
constexpr int kFreeTile = 128, kFreeReach = kFreeMost - 1, kFreeWarps = 32;

__global__ void __launch_bounds__(32 * kFreeWarps) k_free(const uint64_t* __restrict__ bits, int W, int H, int TY,
                                              uint8_t* __restrict__ out) {
    __shared__ uint8_t s_y[kFreeTile + 2 * kFreeReach][32];
    const unsigned yb = ((unsigned)H + 32u) >> 5, bx = blockIdx.x / yb;
    const int x0 = (int)(bx * kFreeTile), lane = threadIdx.x, y = (int)((blockIdx.x - bx * yb) * 32 + lane);
    for (int i = threadIdx.y; i < kFreeTile + 2 * kFreeReach; i += kFreeWarps) {
        const int x = x0 - kFreeReach + i;
        s_y[i][lane] = (uint8_t)(x >= 0 && x < W && y < H ? free_y(bits, TY, x, y) : kFreeMost);
    }
    __syncthreads();
    if (y > H) return;
    for (int j = threadIdx.y; j < kFreeTile && x0 + j <= W; j += kFreeWarps) {
        int d = 1;
        if (x0 + j < W && y < H) {
            d = s_y[j + kFreeReach][lane];
            for (int e = 1; e < d; ++e)
                d = min(d, max(e, (int)min(s_y[j + kFreeReach - e][lane], s_y[j + kFreeReach + e][lane])));
        }
        out[(size_t)(x0 + j) * (H + 1) + y] = (uint8_t)d;
    }
}

inline unsigned blocks_for(long long n, int b) { return (unsigned)((n + b - 1) / b); }

}  // namespace

cudaError_t launch_pack_bits(const uint8_t* d_occ, int W, int H, bool rows, uint64_t* d_bits, cudaStream_t s) {
    int TY = (H + 7) >> 3, TX = (W + 7) >> 3;
    long long n = (long long)TX * TY;
    if (n == 0) return cudaSuccess;
    if (rows) k_pack_bits<true><<<blocks_for(n, 256), 256, 0, s>>>(d_occ, W, H, TY, d_bits);
    else k_pack_bits<false><<<blocks_for(n, 256), 256, 0, s>>>(d_occ, W, H, TY, d_bits);
    return cudaGetLastError();
}

cudaError_t launch_copy_bits(const uint64_t* d_bits, size_t words, uint64_t* out, cudaStream_t s) {
    if (words == 0) return cudaSuccess;
    k_copy_bits<<<min(blocks_for((long long)words, 256), 8u * 152u), 256, 0, s>>>(d_bits, words, out);
    return cudaGetLastError();
}

size_t edt_scratch_bytes(int W, int H) {
    if (W <= kEdtIntSide && H <= kEdtIntSide)   // pass-1 distances and their block minima, uint16
        return ((size_t)W + (size_t)((W + kEdtBlock - 1) / kEdtBlock) + (size_t)((W + kEdtFar - 1) / kEdtFar)) * H *
               sizeof(uint16_t);
    // pass-1 output g (W*H floats) + per-line v (n uint32) and z (n+1 doubles);
    // both passes reuse the same v/z region sized for the larger pass
    size_t g = (size_t)W * H * sizeof(float);
    size_t p1 = (size_t)W * H * sizeof(uint32_t) + (size_t)W * (H + 1) * sizeof(double);
    size_t p2 = (size_t)H * W * sizeof(uint32_t) + (size_t)H * (W + 1) * sizeof(double);
    size_t vz = p1 > p2 ? p1 : p2;
    return ((g + 255) & ~(size_t)255) + vz + 256;
}

cudaError_t launch_edt(const uint64_t* d_bits, int W, int H, int TY, const DtOut& o, void* scratch,
                       size_t scratch_bytes, cudaStream_t s) {
    if (W <= 0 || H <= 0) return cudaSuccess;
    if (scratch_bytes < edt_scratch_bytes(W, H)) return cudaErrorInvalidValue;
    const bool all = o.tiled != nullptr;
    char* base = static_cast<char*>(scratch);
    if (W <= kEdtIntSide && H <= kEdtIntSide) {
        uint16_t* g = reinterpret_cast<uint16_t*>(base);
        uint16_t* gmin = g + (size_t)W * H;
        uint16_t* gfar = gmin + (size_t)((W + kEdtBlock - 1) / kEdtBlock) * H;
        const size_t smem = (size_t)8 * 2 * TY * sizeof(uint16_t);   // at most 64 KB
        static std::atomic<unsigned long long> attr_done{0};
        cudaError_t e = ensure_smem_attr(k_edt_cols, 8 * 2 * (kEdtIntSide / 8) * (int)sizeof(uint16_t), attr_done);
        if (e != cudaSuccess) return e;
        k_edt_cols<<<dim3((W + 7) >> 3, min(4, (H + 255) / 256)), 256, smem, s>>>(d_bits, W, H, TY, g);
        e = cudaGetLastError();
        if (e != cudaSuccess) return e;
        k_edt_block_min<<<dim3(blocks_for(H, 256), (W + kEdtFar - 1) / kEdtFar), 256, 0, s>>>(g, W, H, gmin, gfar);
        e = cudaGetLastError();
        if (e != cudaSuccess) return e;
        const dim3 grid(blocks_for((long long)TY * 8, 32), (W + 7) >> 3), block(32, 8);
        // keys below 2^24 are exact; see above for the bounds of what rounding adds
        const bool exact = (long long)(W - 1) * (W - 1) + (long long)(H - 1) * (H - 1) < (1ll << 24);
        const int slack = exact ? 0 : (W <= kEdtExactSide && H <= kEdtExactSide ? 1 : 24);
        if (exact && all) k_edt_rows<true, true><<<grid, block, 0, s>>>(g, gmin, gfar, W, H, TY, slack, o);
        else if (exact) k_edt_rows<true, false><<<grid, block, 0, s>>>(g, gmin, gfar, W, H, TY, slack, o);
        else if (all) k_edt_rows<false, true><<<grid, block, 0, s>>>(g, gmin, gfar, W, H, TY, slack, o);
        else k_edt_rows<false, false><<<grid, block, 0, s>>>(g, gmin, gfar, W, H, TY, slack, o);
        return cudaGetLastError();
    }
    float* g = reinterpret_cast<float*>(base);
    size_t goff = ((size_t)W * H * sizeof(float) + 255) & ~(size_t)255;
    // per pass: z (n+1 doubles per line) first, then v (n uint32 per line)
    double* z1 = reinterpret_cast<double*>(base + goff);
    uint32_t* v1 = reinterpret_cast<uint32_t*>(base + goff + (size_t)W * (H + 1) * sizeof(double));
    k_edt_pass_y<<<blocks_for(W, 64), 64, 0, s>>>(d_bits, W, H, TY, g, v1, z1);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    double* z2 = reinterpret_cast<double*>(base + goff);
    uint32_t* v2 = reinterpret_cast<uint32_t*>(base + goff + (size_t)H * (W + 1) * sizeof(double));
    k_edt_pass_x<<<blocks_for(H, 64), 64, 0, s>>>(g, W, H, o.dt, v2, z2);
    e = cudaGetLastError();
    if (e != cudaSuccess || !all) return e;
    k_dt_layouts<<<blocks_for((long long)((W + 7) >> 3) * TY * 64, 256), 256, 0, s>>>(o.dt, W, H, TY, o);
    return cudaGetLastError();
}

size_t step_map_cells(int W, int H) {
    const unsigned long long cells = ((unsigned long long)W + 1) * ((unsigned long long)H + 1);
    return cells < (1ull << 32) ? (size_t)cells : 0;
}

size_t step_eq_words(int W, int H) {
    return (size_t)W * ((H + 31) >> 5) + (size_t)((W + 31) >> 5) * H;
}

cudaError_t launch_step_runs(const float* d_step, int W, int H, uint32_t* d_eq, uint32_t* d_runs, unsigned long long* d_share,
                             cudaStream_t s) {
    if ((long long)W * H == 0) return cudaSuccess;
    const int HW = (H + 31) >> 5, XW = (W + 31) >> 5;
    uint32_t* eqy = d_eq;
    uint32_t* eqx = d_eq + (size_t)W * HW;
    k_step_eq<<<blocks_for((long long)XW * HW, 8), 256, 0, s>>>(d_step, W, H, HW, eqx, eqy, d_share);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    k_step_runs<<<blocks_for(H, 32) * blocks_for(W, 8), dim3(32, 8), 0, s>>>(eqx, eqy, d_step, W, H, HW, d_runs, d_share);
    return cudaGetLastError();
}

cudaError_t launch_free_map(const uint64_t* d_bits, int W, int H, int TY, uint8_t* d_free, cudaStream_t s) {
    if ((long long)W * H == 0) return cudaSuccess;
    k_free<<<blocks_for((long long)H + 1, 32) * blocks_for((long long)W + 1, kFreeTile), dim3(32, kFreeWarps), 0, s>>>(
        d_bits, W, H, TY, d_free);
    return cudaGetLastError();
}

cudaError_t launch_edge_map(const uint64_t* d_bits, int W, int H, int TY, uint8_t* d_edge, cudaStream_t s) {
    long long n = (long long)W * H;
    if (n == 0) return cudaSuccess;
    k_edge_map<<<blocks_for(n, 256), 256, 0, s>>>(d_bits, W, H, TY, d_edge);
    return cudaGetLastError();
}

}  // namespace rlc

// ===========================================================================
// rlc_distance_transform_noalloc: the distance transform for callers that
// cannot allocate device memory.
//
// Some callers may not call cudaMalloc at all: real-time loops (a robot's
// localisation node) that forbid allocation after start-up, and hosts whose
// device memory belongs to another allocator (a framework's caching
// allocator, a fixed pool handed out by an embedding application).  This
// entry point computes the same distance transform as
// rlc_map_distance_transform from a caller-owned device occupancy grid into
// a caller-owned device output, and keeps every intermediate (the packed
// occupancy bits, the first-pass output and the per-line envelope arrays) in
// one file-scope device array of fixed size, so it allocates nothing.
//
// * The array holds RLC_NOALLOC_SCRATCH_BYTES (~16.2 MiB) on every GPU that
//   loads this library, until the process exits.
// * Maps are limited to RLC_NOALLOC_MAX_CELLS cells with sides of at most
//   RLC_NOALLOC_MAX_SIDE; larger maps are rejected with RLC_ERR_ARG.
// * The first call on a device looks up the array's device address there
//   (cudaGetSymbolAddress, with that device current) and caches it; make
//   that first call before any stream capture.  The cached address lives as
//   long as the device's primary context: after cudaDeviceReset the library
//   has to be unloaded and loaded again before this entry point is used.
// * All calls share the array and it keeps the last call's contents.  No
//   word of it needs to start at zero (each is written before it is read),
//   but calls that overlap on the GPU -- on different streams, or from
//   different host threads -- race on it and corrupt each other's results.
// ===========================================================================
namespace rlc {
namespace {

constexpr size_t align_up(size_t b) { return (b + 255) & ~(size_t)255; }
constexpr size_t kNoAllocMaxCells = RLC_NOALLOC_MAX_CELLS;
constexpr size_t kNoAllocMaxSide = RLC_NOALLOC_MAX_SIDE;
// packed bits: ceil(W/8) * ceil(H/8) words <= cells/64 + (W + H)/8 + 1
constexpr size_t kNoAllocBitsBytes = align_up((kNoAllocMaxCells / 64 + 2 * kNoAllocMaxSide / 8 + 1) * 8);
constexpr size_t kNoAllocScratchBytes = kNoAllocBitsBytes + edt_scratch_bound(kNoAllocMaxCells, kNoAllocMaxSide);
static_assert(kNoAllocScratchBytes == RLC_NOALLOC_SCRATCH_BYTES, "rangelibc.h states the scratch size");

static __device__ __align__(256) unsigned char g_noalloc_scratch[kNoAllocScratchBytes];

constexpr int kMaxDevices = 64;
std::mutex g_noalloc_mu;
void* g_noalloc_addr[kMaxDevices] = {};

// device address of g_noalloc_scratch on the current device (looked up once per device)
int noalloc_scratch(void** out) {
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    char msg[256];
    if (e != cudaSuccess) {
        snprintf(msg, sizeof(msg), "rlc_distance_transform_noalloc: %s", cudaGetErrorString(e));
        return set_last_error(RLC_ERR_CUDA, msg);
    }
    if (dev < 0 || dev >= kMaxDevices) return set_last_error(RLC_ERR_CUDA, "rlc_distance_transform_noalloc: device ordinal out of range");
    std::lock_guard<std::mutex> lk(g_noalloc_mu);
    if (!g_noalloc_addr[dev]) {
        void* p = nullptr;
        e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
        if (e != cudaSuccess || !p) {
            snprintf(msg, sizeof(msg), "rlc_distance_transform_noalloc: scratch address: %s",
                     cudaGetErrorString(e));
            return set_last_error(RLC_ERR_CUDA, msg);
        }
        g_noalloc_addr[dev] = p;
    }
    *out = g_noalloc_addr[dev];
    return RLC_OK;
}

// device memory of the current device, or managed memory; memory of another device is refused
// (without peer access the kernels here would fault on it)
bool is_device_pointer(const void* p) {
    cudaPointerAttributes a;
    if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    if (a.type == cudaMemoryTypeManaged) return true;
    if (a.type != cudaMemoryTypeDevice) return false;
    int dev = -1;
    if (cudaGetDevice(&dev) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    return a.device == dev;
}

}  // namespace
}  // namespace rlc

extern "C" int rlc_distance_transform_noalloc(const uint8_t* d_occ, int width, int height, float* d_dt,
                                              void* stream) {
    using namespace rlc;
    char msg[256];
    if (!d_occ || !d_dt) return set_last_error(RLC_ERR_ARG, "rlc_distance_transform_noalloc: null pointer");
    if (width <= 0 || height <= 0) return set_last_error(RLC_ERR_ARG, "rlc_distance_transform_noalloc: sizes must be positive");
    if ((size_t)width > kNoAllocMaxSide || (size_t)height > kNoAllocMaxSide ||
        (size_t)width * (size_t)height > kNoAllocMaxCells) {
        snprintf(msg, sizeof(msg),
                 "rlc_distance_transform_noalloc: a %dx%d map exceeds the fixed scratch (at most %zu cells and "
                 "%zu per side); use rlc_map_create + rlc_map_distance_transform",
                 width, height, kNoAllocMaxCells, kNoAllocMaxSide);
        return set_last_error(RLC_ERR_ARG, msg);
    }
    if (!is_device_pointer(d_occ) || !is_device_pointer(d_dt))
        return set_last_error(RLC_ERR_ARG, "rlc_distance_transform_noalloc: d_occ and d_dt must be device memory of the current device");
    void* base = nullptr;
    if (int rc = noalloc_scratch(&base)) return rc;
    cudaStream_t s = (cudaStream_t)stream;
    uint64_t* bits = static_cast<uint64_t*>(base);
    void* edt_scratch = static_cast<char*>(base) + kNoAllocBitsBytes;
    const int TY = (height + 7) >> 3;
    cudaError_t e = launch_pack_bits(d_occ, width, height, false, bits, s);
    if (e == cudaSuccess)
        e = launch_edt(bits, width, height, TY, DtOut{d_dt}, edt_scratch, kNoAllocScratchBytes - kNoAllocBitsBytes, s);
    if (e != cudaSuccess) {
        snprintf(msg, sizeof(msg), "rlc_distance_transform_noalloc: %s", cudaGetErrorString(e));
        return set_last_error(RLC_ERR_CUDA, msg);
    }
    return RLC_OK;
}
