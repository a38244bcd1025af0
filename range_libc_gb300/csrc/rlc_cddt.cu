// CDDT (compressed directional distance transform) table, built and pruned
// on the device, plus the scan primitive it uses.
//
// The table follows the reference's construction (RangeLib.h:974-1159):
// for every edge pixel and every slice a < td/2, the pixel centre is
// projected into the slice's rotated frame and its x coordinate is appended
// to each bin its y extent covers; every bin is then sorted and
// de-duplicated.  Prune (RangeLib.h:1176-1283) replays a query from every
// free cell centre of every slice and keeps only the zero points a query can
// return.  Here those steps are: a list of the edge pixels, a count pass and a
// fill pass (a block per slice and chunk of edge pixels, the slice's bins in
// shared memory), an exclusive scan to CSR offsets, a sort of every bin with
// de-duplication (a warp per bin in registers), and a final compaction;
// prune marks used entries with one thread per (cell, slice)
// and compacts with the same scan.
//
// Device layout: slice a owns bins [slice_base[a], slice_base[a+1]); bin b
// owns zeros [bin_start[b], bin_start[b+1]).  All offsets are uint32.
#include "rlc_internal.cuh"

#include <algorithm>
#include <cmath>
#include <cstdio>
#include <vector>

namespace rlc {
namespace {

constexpr double kEps = 0.00001;   // RangeLib.h:60 _EPSILON
constexpr int kBinarySearchThreshold = 64;

inline unsigned blocks_for(long long n, int b) { return (unsigned)((n + b - 1) / b); }

// ------------------------------------------------------------------- scan
constexpr int kScanThreads = 512;
constexpr int kScanItems = 8;
constexpr int kScanTile = kScanThreads * kScanItems;

struct OpSum {
    typedef uint32_t T;
    static __device__ __forceinline__ T id() { return 0u; }
    static __device__ __forceinline__ T op(T a, T b) { return a + b; }
};
struct OpMax {
    typedef int T;
    static __device__ __forceinline__ T id() { return -2147483647 - 1; }
    static __device__ __forceinline__ T op(T a, T b) { return a > b ? a : b; }
};

// block-wide scan of one value per thread: returns the exclusive prefix,
// `total` gets the reduction over the block
template <class Op>
__device__ __forceinline__ typename Op::T block_scan(typename Op::T v, typename Op::T* warp_vals,
                                                     typename Op::T& total) {
    typedef typename Op::T T;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    T x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        T y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x = Op::op(y, x);
    }
    T excl_in_warp = __shfl_up_sync(0xffffffffu, x, 1);
    if (lane == 0) excl_in_warp = Op::id();
    if (lane == 31) warp_vals[wid] = x;
    __syncthreads();
    if (wid == 0) {
        const int nw = blockDim.x >> 5;
        T w = lane < nw ? warp_vals[lane] : Op::id();
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            T y = __shfl_up_sync(0xffffffffu, w, o);
            if (lane >= o) w = Op::op(y, w);
        }
        if (lane < nw) warp_vals[lane] = w;
    }
    __syncthreads();
    total = warp_vals[(blockDim.x >> 5) - 1];
    T excl = wid > 0 ? Op::op(warp_vals[wid - 1], excl_in_warp) : excl_in_warp;
    __syncthreads();
    return excl;
}

template <class Op>
__global__ void __launch_bounds__(kScanThreads) k_tile_reduce(const typename Op::T* __restrict__ in, size_t n,
                                                              typename Op::T* __restrict__ sums) {
    __shared__ typename Op::T ws[32];
    size_t base = (size_t)blockIdx.x * kScanTile + (size_t)threadIdx.x * kScanItems;
    typename Op::T s = Op::id();
#pragma unroll
    for (int i = 0; i < kScanItems; ++i)
        if (base + i < n) s = Op::op(s, in[base + i]);
    typename Op::T total;
    block_scan<Op>(s, ws, total);
    if (threadIdx.x == 0) sums[blockIdx.x] = total;
}

// single block: exclusive scan of the tile reductions in place; sums[ntiles] = total
template <class Op>
__global__ void __launch_bounds__(kScanThreads) k_scan_partials(typename Op::T* sums, size_t ntiles) {
    __shared__ typename Op::T ws[32];
    typename Op::T carry = Op::id();
    for (size_t base = 0; base < ntiles; base += kScanThreads) {
        size_t i = base + threadIdx.x;
        typename Op::T v = i < ntiles ? sums[i] : Op::id();
        typename Op::T total;
        typename Op::T e = block_scan<Op>(v, ws, total);
        if (i < ntiles) sums[i] = Op::op(carry, e);
        carry = Op::op(carry, total);
    }
    if (threadIdx.x == 0) sums[ntiles] = carry;
}

// INCLUSIVE = false: out[i] = op(in[0..i-1]) and out[n] = total; true: out[i] = op(in[0..i])
template <class Op, bool INCLUSIVE>
__global__ void __launch_bounds__(kScanThreads) k_scan_tiles(const typename Op::T* __restrict__ in, size_t n,
                                                             const typename Op::T* __restrict__ sums,
                                                             typename Op::T* __restrict__ out, size_t ntiles) {
    typedef typename Op::T T;
    __shared__ T ws[32];
    size_t base = (size_t)blockIdx.x * kScanTile + (size_t)threadIdx.x * kScanItems;
    T v[kScanItems];
    T s = Op::id();
#pragma unroll
    for (int i = 0; i < kScanItems; ++i) {
        v[i] = base + i < n ? in[base + i] : Op::id();
        s = Op::op(s, v[i]);
    }
    T total;
    T run = Op::op(sums[blockIdx.x], block_scan<Op>(s, ws, total));
#pragma unroll
    for (int i = 0; i < kScanItems; ++i) {
        if (INCLUSIVE) run = Op::op(run, v[i]);
        if (base + i < n) out[base + i] = run;
        if (!INCLUSIVE) run = Op::op(run, v[i]);
    }
    if (!INCLUSIVE && blockIdx.x == 0 && threadIdx.x == 0) out[n] = sums[ntiles];
}

// ------------------------------------------------------------ construction
__device__ __forceinline__ bool occ_bit(const uint64_t* __restrict__ bits, int TY, int x, int y) {
    uint64_t w = __ldg(bits + (size_t)(x >> 3) * TY + (y >> 3));
    return (w >> (((x & 7) << 3) | (y & 7))) & 1ull;
}

struct SliceGeom {
    const int* widths;
    const float* trans;
    const float* cosv;
    const float* sinv;
    const uint32_t* slice_base;
};

// (int)(v + eps) or (int)(v - eps) in double.  Where v is not negative and its fraction (exact in float)
// is not near eps or 1 - eps, whole and fraction decide: the six double steps of a projection would hold
// the FP64 pipe for about 90 us on the 7.2 M projections of a 2048 x 2048 map.
template <bool PLUS>
__device__ __forceinline__ int trunc_off(float v) {
    const int whole = __float2int_rz(v);
    const float frac = __fsub_rn(v, __int2float_rn(whole));
    const float d = PLUS ? __fsub_rn(1.0f, frac) : frac;   // eps or more of this: no carry
    if (v >= 0.0f && v < 8388608.0f && !(d > 0.9e-5f && d < 1.1e-5f))
        return d >= 1e-5f || (!PLUS && whole == 0) ? whole : (PLUS ? whole + 1 : whole - 1);
    return __double2int_rz(PLUS ? __dadd_rn((double)v, kEps) : __dsub_rn((double)v, kEps));
}

// RangeLib.h:1086-1103: projection of a pixel centre into slice a.
__device__ __forceinline__ void project_pixel(const SliceGeom& g, int a, int x, int y, float& lcx, int& lower,
                                              int& upper) {
    const float ca = __ldg(g.cosv + a), sa = __ldg(g.sinv + a);
    const float half = __fmul_rn(__fadd_rn(fabsf(sa), fabsf(ca)), 0.5f);   // (|s|+|c|) / 2.0, exact halving
    const float px = __int2float_rn(x) + 0.5f, py = __int2float_rn(y) + 0.5f;   // exact for grids < 2^23
    lcx = __fsub_rn(__fmul_rn(px, ca), __fmul_rn(py, sa));
    const float lcy = __fadd_rn(__fadd_rn(__fmul_rn(px, sa), __fmul_rn(py, ca)), __ldg(g.trans + a));
    const float top = __fadd_rn(lcy, half), bottom = __fsub_rn(lcy, half);
    upper = trunc_off<false>(top);
    lower = trunc_off<true>(bottom);
}

// Edge pixels: occupied with a free neighbour in the grid; a thread per 8 x 8 word of the map, its
// neighbours' free bits moved over its own.  *n counts them; with `edges` (room for all) they are listed,
// in no order.
// the cells of word (tx, ty) that lie in the grid
__device__ __forceinline__ uint64_t grid_word(int W, int H, int tx, int ty) {
    uint64_t in = ~0ull;
    if (8 * tx + 8 > W) in = (1ull << (8 * (W - 8 * tx))) - 1ull;
    if (8 * ty + 8 > H) in &= 0x0101010101010101ull * ((1u << (H - 8 * ty)) - 1u);
    return in;
}

__device__ __forceinline__ uint64_t free_word(const uint64_t* __restrict__ bits, int W, int H, int TX, int TY, int tx, int ty) {
    if (tx < 0 || ty < 0 || tx >= TX || ty >= TY) return 0ull;
    return ~__ldg(bits + (size_t)tx * TY + ty) & grid_word(W, H, tx, ty);
}

__global__ void __launch_bounds__(256) k_edges(const uint64_t* __restrict__ bits, int W, int H, int TX, int TY,
                                               uint32_t* __restrict__ edges, uint32_t* __restrict__ n) {
    __shared__ uint32_t s_sum[8], s_base;
    const uint64_t low = 0x0101010101010101ull;
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const int tx = (int)(i / TY), ty = (int)(i - (long long)tx * TY);
    uint64_t edge = 0ull;
    if (i < (long long)TX * TY) {
        uint64_t v[3];   // free in the column before, of and after each cell, per word along y
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            const uint64_t a = free_word(bits, W, H, TX, TY, tx - 1, ty + k - 1), c = free_word(bits, W, H, TX, TY, tx, ty + k - 1),
                           b = free_word(bits, W, H, TX, TY, tx + 1, ty + k - 1);
            v[k] = c | (c << 8) | (a >> 56) | (c >> 8) | (b << 56);
        }
        const uint64_t near = v[1] | ((v[1] & ~(low << 7)) << 1) | ((v[1] >> 1) & ~(low << 7)) | ((v[0] >> 7) & low) | ((v[2] & low) << 7);
        edge = __ldg(bits + i) & grid_word(W, H, tx, ty) & near;
    }
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const uint32_t mine = (uint32_t)__popcll(edge);
    uint32_t at = mine;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t t = __shfl_up_sync(0xffffffffu, at, o);
        if (lane >= o) at += t;
    }
    if (lane == 31) s_sum[wid] = at;
    __syncthreads();
    if (threadIdx.x == 0) {
        uint32_t sum = 0;
        for (int w = 0; w < 8; ++w) {
            const uint32_t t = s_sum[w];
            s_sum[w] = sum;
            sum += t;
        }
        s_base = sum ? atomicAdd(n, sum) : 0u;
    }
    __syncthreads();
    if (!edges) return;
    at += s_base + s_sum[wid] - mine;
    while (edge) {
        const int bit = __ffsll((long long)edge) - 1;
        edge &= edge - 1;
        edges[at++] = (uint32_t)(8 * tx + (bit >> 3)) * (uint32_t)H + (uint32_t)(8 * ty + (bit & 7));
    }
}

// pass 0 counts entries per bin, pass 1 scatters them
template <int PASS>
__global__ void k_project(SliceGeom g, const uint32_t* __restrict__ edges, uint32_t nedges, int H, int nslices,
                          uint32_t* __restrict__ counts, const uint32_t* __restrict__ start,
                          float* __restrict__ zeros) {
    long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= (long long)nedges * nslices) return;
    int a = (int)(t % nslices);
    uint32_t cell = __ldg(edges + t / nslices);
    int x = (int)(cell / (uint32_t)H), y = (int)(cell - (uint32_t)x * (uint32_t)H);
    float lcx;
    int lower, upper;
    project_pixel(g, a, x, y, lcx, lower, upper);
    const int width = __ldg(g.widths + a);
    const uint32_t sb = __ldg(g.slice_base + a);
    for (int i = lower; i <= upper; ++i) {
        if (i < 0 || i >= width) continue;   // outside the slice (cannot happen for in-grid pixels)
        uint32_t b = sb + (uint32_t)i;
        if (PASS == 0) atomicAdd(counts + b, 1u);
        else zeros[__ldg(start + b) + atomicAdd(counts + b, 1u)] = lcx;
    }
}

// The same with the slice's bins in shared memory: a block per slice and kProjectChunk edge pixels, whose
// entries mostly share bins.  Counting and filling entry by entry in memory took 159 and 249 us for the
// 7.2 M projections of a 2048 x 2048 map with 108 slices, now 88 and 177.
constexpr int kProjectChunk = 8192, kProjectThreads = 512;
constexpr size_t kProjectSmem = 100 * 1024;   // leaves an SM room for a second block

template <int PASS>
__global__ void __launch_bounds__(kProjectThreads) k_project_block(SliceGeom g, const uint32_t* __restrict__ edges,
                                                                   uint32_t nedges, int H, uint32_t* __restrict__ counts,
                                                                   const uint32_t* __restrict__ start,
                                                                   float* __restrict__ zeros) {
    extern __shared__ uint32_t s_bin[];
    const int a = blockIdx.y, width = __ldg(g.widths + a);
    const uint32_t sb = __ldg(g.slice_base + a);
    const uint32_t e0 = blockIdx.x * (uint32_t)kProjectChunk, e1 = min(e0 + (uint32_t)kProjectChunk, nedges);
    for (int i = threadIdx.x; i < width; i += kProjectThreads) s_bin[i] = 0u;
    __syncthreads();
    auto each = [&](auto f) {
        for (uint32_t e = e0 + threadIdx.x; e < e1; e += kProjectThreads) {
            const uint32_t cell = __ldg(edges + e);
            const int x = (int)(cell / (uint32_t)H), y = (int)(cell - (uint32_t)x * (uint32_t)H);
            float lcx;
            int lower, upper;
            project_pixel(g, a, x, y, lcx, lower, upper);
            for (int i = max(lower, 0); i <= min(upper, width - 1); ++i) f(i, lcx);
        }
    };
    each([&](int i, float) { atomicAdd(s_bin + i, 1u); });
    __syncthreads();
    for (int i = threadIdx.x; i < width; i += kProjectThreads)
        if (s_bin[i]) {
            const uint32_t before = atomicAdd(counts + sb + i, s_bin[i]);
            if (PASS == 1) s_bin[i] = __ldg(start + sb + i) + before;   // this block's places in the bin
        }
    if (PASS == 1) {
        __syncthreads();
        each([&](int i, float lcx) { zeros[atomicAdd(s_bin + i, 1u)] = lcx; });
    }
}

// out[0] = the largest count, out[1] = their sum
__global__ void k_count_stats(const uint32_t* __restrict__ v, size_t n, unsigned long long* out) {
    unsigned long long m = 0, sum = 0;
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
        m = max(m, (unsigned long long)v[i]);
        sum += v[i];
    }
    for (int o = 16; o; o >>= 1) {
        m = max(m, __shfl_xor_sync(0xffffffffu, m, o));
        sum += __shfl_xor_sync(0xffffffffu, sum, o);
    }
    if ((threadIdx.x & 31) == 0) {
        atomicMax(out, m);
        atomicAdd(out + 1, sum);
    }
}

// Bins of up to 32 R entries: a warp sorts its bin in registers (entry R * lane + r, bitonic) and writes the
// distinct values in place; ucount[b] receives their number.  Longer ones are listed for k_sort_unique.
// A block per bin with one thread de-duplicating took 1.08 ms for the 281,593 bins of that map, now 0.41 and 0.11 for the listed ones.
template <int R>
__device__ __forceinline__ void sort_bin(float* z, int n, int lane, uint32_t* ucount) {
    const float inf = __int_as_float(0x7f800000);
    float v[R];
#pragma unroll
    for (int r = 0; r < R; ++r) v[r] = r * 32 + lane < n ? z[r * 32 + lane] : inf;
#pragma unroll
    for (int k = 2; k <= 32 * R; k <<= 1)
#pragma unroll
        for (int j = k >> 1; j > 0; j >>= 1)
            if (j >= R) {
#pragma unroll
                for (int r = 0; r < R; ++r) {
                    const float o = __shfl_xor_sync(0xffffffffu, v[r], j / R);
                    const int i = lane * R + r;
                    const bool low = ((i & j) == 0) == ((i & k) == 0);   // keeps the smaller of the two
                    v[r] = (low ? o < v[r] : v[r] < o) ? o : v[r];
                }
            } else {
#pragma unroll
                for (int r = 0; r < R; ++r)
                    if (!(r & j)) {
                        const bool up = ((lane * R + r) & k) == 0;
                        const float x = v[r], y = v[r | j];
                        const bool swap = up ? y < x : x < y;
                        v[r] = swap ? y : x;
                        v[r | j] = swap ? x : y;
                    }
            }
    // distinct values, in order
    const float before = __shfl_up_sync(0xffffffffu, v[R - 1], 1);
    int keep = 0;
    bool first[R];
#pragma unroll
    for (int r = 0; r < R; ++r) {
        const int i = lane * R + r;
        first[r] = i < n && (i == 0 || v[r] != (r ? v[r - 1] : before));
        keep += first[r];
    }
    int at = keep;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int t = __shfl_up_sync(0xffffffffu, at, o);
        if (lane >= o) at += t;
    }
    if (lane == 31) *ucount = (uint32_t)at;
    at -= keep;
#pragma unroll
    for (int r = 0; r < R; ++r)
        if (first[r]) z[at++] = v[r];
}

__global__ void __launch_bounds__(256) k_sort_bins(const uint32_t* __restrict__ start, uint32_t nb, float* zeros,
                                                   uint32_t* __restrict__ ucount, uint32_t* __restrict__ longer) {
    const uint32_t b = blockIdx.x * 8u + (threadIdx.x >> 5);
    const int lane = threadIdx.x & 31;
    if (b >= nb) return;
    const uint32_t lo = __ldg(start + b);
    const int n = (int)(__ldg(start + b + 1) - lo);
    if (n == 0) {
        if (lane == 0) ucount[b] = 0u;
    } else if (n <= 32) {
        sort_bin<1>(zeros + lo, n, lane, ucount + b);
    } else if (n <= 64) {
        sort_bin<2>(zeros + lo, n, lane, ucount + b);
    } else if (n <= 128) {
        sort_bin<4>(zeros + lo, n, lane, ucount + b);
    } else if (n <= 256) {
        sort_bin<8>(zeros + lo, n, lane, ucount + b);
    } else if (lane == 0) {
        longer[1 + atomicAdd(longer, 1u)] = b;
    }
}

constexpr size_t kSortSmem = 200 * 1024;

// the listed bins, a block each: bitonic sort in shared memory, then de-duplicate in
// place; ucount[b] receives the number of distinct values
__device__ void sort_unique_block(uint32_t b, const uint32_t* __restrict__ start, float* zeros, uint32_t* __restrict__ ucount, float* sh) {
    const uint32_t lo = start[b];
    const int n = (int)(start[b + 1] - lo);
    int p = 1;
    while (p < n) p <<= 1;
    for (int i = threadIdx.x; i < p; i += blockDim.x) sh[i] = i < n ? zeros[lo + i] : __int_as_float(0x7f800000);
    __syncthreads();
    for (int k = 2; k <= p; k <<= 1) {
        for (int j = k >> 1; j > 0; j >>= 1) {
            for (int i = threadIdx.x; i < p; i += blockDim.x) {
                int l = i ^ j;
                if (l > i) {
                    float a = sh[i], c = sh[l];
                    bool up = (i & k) == 0;
                    if (up ? (c < a) : (a < c)) { sh[i] = c; sh[l] = a; }
                }
            }
            __syncthreads();
        }
    }
    // distinct values, 32 at a time by the first warp
    if (threadIdx.x < 32) {
        const int lane = threadIdx.x;
        int w = 0;
        for (int i0 = 0; i0 < n; i0 += 32) {
            const int i = i0 + lane;
            const bool first = i < n && (i == 0 || sh[i] != sh[i - 1]);
            const unsigned who = __ballot_sync(0xffffffffu, first);
            if (first) zeros[lo + w + __popc(who & ((1u << lane) - 1u))] = sh[i];
            w += __popc(who);
        }
        if (lane == 0) ucount[b] = (uint32_t)w;
    }
    __syncthreads();
}

__global__ void __launch_bounds__(256) k_sort_unique(const uint32_t* __restrict__ longer, const uint32_t* __restrict__ start,
                                                     float* zeros, uint32_t* __restrict__ ucount) {
    extern __shared__ float sh[];
    const uint32_t n = longer[0];
    for (uint32_t i = blockIdx.x; i < n; i += gridDim.x) sort_unique_block(longer[1 + i], start, zeros, ucount, sh);
}

// a warp per bin
__global__ void __launch_bounds__(256) k_copy_bins(const uint32_t* __restrict__ src_start, const float* __restrict__ src,
                                                   uint32_t nb, const uint32_t* __restrict__ dst_start,
                                                   float* __restrict__ dst) {
    const uint32_t b = blockIdx.x * 8u + (threadIdx.x >> 5);
    if (b >= nb) return;
    const uint32_t s = __ldg(src_start + b), d = __ldg(dst_start + b), n = __ldg(dst_start + b + 1) - d;
    for (uint32_t i = threadIdx.x & 31; i < n; i += 32) dst[d + i] = __ldg(src + s + i);
}

// ------------------------------------------------------------------ prune
// One slice per launch, one thread per cell in the reference's visiting
// order (cell = x * H + y).  A cell either skips, marks directly, or -- in
// the linear-search branch when no zero point is >= x -- reuses the index
// the last assigning cell of the slice produced (the reference leaves its
// `index` unassigned there, RangeLib.h:1242-1247, and keeps the stale value).
// tag[c] = c for cells that assign an index (val[c] = that index), -1 for
// cells that do not, and -2 for cells that need the stale index.
__global__ void k_prune_classify(SliceGeom g, int a, const uint64_t* __restrict__ bits, int W, int H, int TY,
                                 const uint32_t* __restrict__ bin_start, const float* __restrict__ zeros, float mr,
                                 uint32_t* __restrict__ used, int* __restrict__ tag, int* __restrict__ val,
                                 unsigned* __restrict__ n_need) {
    const long long ncell = (long long)W * H;
    const long long c = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= ncell) return;
    const float ca = __ldg(g.cosv + a), sa = __ldg(g.sinv + a), tr = __ldg(g.trans + a);
    int x = (int)(c / H), y = (int)(c - (long long)x * H);
    int t = -1;
    const float fx = __int2float_rn(x) + 0.5f, fy = __int2float_rn(y) + 0.5f;
    const float lx = __fsub_rn(__fmul_rn(fx, ca), __fmul_rn(fy, sa));
    const float ly = __fadd_rn(__fadd_rn(__fmul_rn(fx, sa), __fmul_rn(fy, ca)), tr);
    const unsigned li = (unsigned)__float2int_rz(ly);
    if (li < (unsigned)__ldg(g.widths + a)) {
        const uint32_t b = __ldg(g.slice_base + a) + li;
        const uint32_t base = __ldg(bin_start + b);
        const int n = (int)(__ldg(bin_start + b + 1) - base);
        const int high = n - 1;
        if (high >= 0 && !occ_bit(bits, TY, x, y)) {
            const float last = __ldg(zeros + base + high);
            if (last < lx && __fsub_rn(lx, last) < mr) {
                used[base + high] = 1;
            } else {
                int index = -1;
                if (high > kBinarySearchThreshold) {
                    int l = 0, h = n;   // lower_bound
                    while (l < h) {
                        int mid = (l + h) >> 1;
                        if (__ldg(zeros + base + mid) < lx) l = mid + 1; else h = mid;
                    }
                    index = l;
                } else {
                    for (int i = 0; i < n; ++i)
                        if (__ldg(zeros + base + i) >= lx) { index = i; break; }
                }
                if (index >= 0) {
                    if (index < n) used[base + index] = 1;
                    if (index >= 1) used[base + index - 1] = 1;
                    t = (int)c;
                    val[c] = index;
                } else {
                    t = -2;
                    atomicAdd(n_need, 1u);
                }
            }
        }
    }
    tag[c] = t;
}

// cells that need the stale index: last[c] is the last assigning cell <= c
__global__ void k_prune_stale(SliceGeom g, int a, int W, int H, const uint32_t* __restrict__ bin_start,
                              const int* __restrict__ tag, const int* __restrict__ last, const int* __restrict__ val,
                              uint32_t* __restrict__ used) {
    const long long ncell = (long long)W * H;
    const long long c = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= ncell || tag[c] != -2) return;
    const int p = last[c];
    const int index = p >= 0 ? val[p] : 0;   // the reference's index starts each slice at 0 here
    int x = (int)(c / H), y = (int)(c - (long long)x * H);
    const float ca = __ldg(g.cosv + a), sa = __ldg(g.sinv + a), tr = __ldg(g.trans + a);
    const float fx = __int2float_rn(x) + 0.5f, fy = __int2float_rn(y) + 0.5f;
    const float ly = __fadd_rn(__fadd_rn(__fmul_rn(fx, sa), __fmul_rn(fy, ca)), tr);
    const unsigned li = (unsigned)__float2int_rz(ly);
    const uint32_t b = __ldg(g.slice_base + a) + li;
    const uint32_t base = __ldg(bin_start + b);
    const int n = (int)(__ldg(bin_start + b + 1) - base);
    if (index >= 0 && index < n) used[base + index] = 1;
    if (index - 1 >= 0 && index - 1 < n) used[base + index - 1] = 1;
}

// entries of slices >= nslices are kept (they are empty after construction)
__global__ void k_keep_flags(uint32_t* __restrict__ used, uint32_t first_unpruned_entry, uint32_t n) {
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n && i >= first_unpruned_entry) used[i] = 1;
}

__global__ void k_compact_entries(const uint32_t* __restrict__ keep, const uint32_t* __restrict__ pos, uint32_t n,
                                  const float* __restrict__ src, float* __restrict__ dst) {
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n && keep[i]) dst[pos[i]] = src[i];
}

__global__ void k_remap_starts(const uint32_t* __restrict__ old_start, const uint32_t* __restrict__ pos,
                               uint32_t nb, uint32_t* __restrict__ new_start) {
    uint32_t b = blockIdx.x * blockDim.x + threadIdx.x;
    if (b <= nb) new_start[b] = pos[old_start[b]];
}

// ------------------------------------------------------------------ index
// one warp per bin: its zero points after -inf and before +inf, in whole quads, and for every bucket k of its slice where
// the zero points with a bucket >= k begin; *bad is set by zero points that are not finite and sorted
struct IndexSlice {   // CddtDev::slices
    float c, s, trans, v0;
    uint32_t width, base, row, unused;
};

// first quad of bin b: at least n + 2 values before the next bin's
__device__ __forceinline__ size_t index_quad(const uint32_t* start, uint32_t b) { return (size_t)(start[b] >> 2) + 2 * (size_t)b; }

__global__ void __launch_bounds__(256) k_index_fill(const IndexSlice* __restrict__ sl,
                                                    const uint32_t* __restrict__ slice_base, int td, uint32_t nb,
                                                    const uint32_t* __restrict__ start, const float* __restrict__ zeros,
                                                    float* __restrict__ qz, uint32_t* __restrict__ index,
                                                    unsigned* __restrict__ bad) {
    const uint32_t b = (uint32_t)(((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5);
    const int lane = threadIdx.x & 31;
    if (b >= nb) return;
    const uint32_t lo = start[b], n = start[b + 1] - lo;
    const float* z = zeros + lo;
    const size_t q0 = index_quad(start, b) * 4, q1 = index_quad(start, b + 1) * 4;
    float* q = qz + q0;
    const float inf = __int_as_float(0x7f800000);
    bool ok = true;
    for (uint32_t i = lane; i < (uint32_t)(q1 - q0); i += 32) {
        float v = i == 0 ? -inf : inf;
        if (i >= 1 && i <= n) {
            v = z[i - 1];
            ok = ok && isfinite(v) && (i == 1 || z[i - 2] <= v);
        }
        q[i] = v;
    }
    if (!ok) *bad = 1u;
    int s0 = 0, s1 = td - 1;   // the bin's slice: the last with slice_base <= b
    while (s0 < s1) {
        const int mid = (s0 + s1 + 1) >> 1;
        if (slice_base[mid] <= b) s0 = mid; else s1 = mid - 1;
    }
    const IndexSlice S = sl[s0];
    for (uint32_t k = lane; k < S.row; k += 32) {
        uint32_t i = 0, e = n;
        if (k + 1 == S.row) i = n;   // the end: the upper sentinel
        else
            while (i < e) {   // first zero point whose bucket is >= k (the last bucket holds what lies beyond)
                const uint32_t mid = (i + e) >> 1;
                const int bk = min(max(cddt_bucket(z[mid], S.v0), 0), (int)S.row - 2);
                if (bk >= (int)k) e = mid; else i = mid + 1;
            }
        index[S.base + (size_t)(b - slice_base[s0]) * S.row + k] = (uint32_t)q0 + 1 + i;
    }
}

__global__ void k_gather_u32(const uint32_t* __restrict__ v, const uint32_t* __restrict__ at, uint32_t n,
                             uint32_t* __restrict__ out) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) out[i] = v[at[i]];
}

struct DevBuf {
    void* p = nullptr;
    ~DevBuf() { if (p) cudaFree(p); }
    cudaError_t alloc(size_t bytes) { return cudaMalloc(&p, bytes ? bytes : 4); }
    template <class T> T* as() const { return static_cast<T*>(p); }
};

#define RLC_TRY(x) do { cudaError_t _e = (x); if (_e != cudaSuccess) return _e; } while (0)

}  // namespace

template <class Op, bool INCLUSIVE>
static cudaError_t scan_impl(const typename Op::T* d_in, typename Op::T* d_out, size_t n, cudaStream_t s) {
    size_t ntiles = (n + kScanTile - 1) / kScanTile;
    if (ntiles == 0) ntiles = 1;
    DevBuf sums;
    RLC_TRY(sums.alloc((ntiles + 1) * sizeof(typename Op::T)));
    k_tile_reduce<Op><<<(unsigned)ntiles, kScanThreads, 0, s>>>(d_in, n, sums.as<typename Op::T>());
    RLC_TRY(cudaGetLastError());
    k_scan_partials<Op><<<1, kScanThreads, 0, s>>>(sums.as<typename Op::T>(), ntiles);
    RLC_TRY(cudaGetLastError());
    k_scan_tiles<Op, INCLUSIVE><<<(unsigned)ntiles, kScanThreads, 0, s>>>(d_in, n, sums.as<typename Op::T>(), d_out,
                                                                         ntiles);
    RLC_TRY(cudaGetLastError());
    return cudaStreamSynchronize(s);   // the temporary is released on return
}

cudaError_t scan_exclusive_u32(const uint32_t* d_in, uint32_t* d_out, size_t n, cudaStream_t s) {
    return scan_impl<OpSum, false>(d_in, d_out, n, s);
}

cudaError_t cddt_build(const uint64_t* d_bits, int W, int H, int TY, unsigned td, const int* d_widths,
                       const float* d_trans, const float* d_cos, const float* d_sin, const uint32_t* h_slice_base,
                       CddtBuild* out, cudaStream_t s, char* why, size_t why_len) {
    const int nslices = (int)((td + 1) / 2);   // a < td / 2.0
    const uint32_t nb = h_slice_base[td];
    const long long ncell = (long long)W * H;
    SliceGeom g{d_widths, d_trans, d_cos, d_sin, nullptr};

    DevBuf slice_base;
    RLC_TRY(slice_base.alloc((td + 1) * sizeof(uint32_t)));
    RLC_TRY(cudaMemcpyAsync(slice_base.p, h_slice_base, (td + 1) * sizeof(uint32_t), cudaMemcpyHostToDevice, s));
    g.slice_base = slice_base.as<uint32_t>();

    // 1. edge pixels
    const int TX = (W + 7) / 8;
    const unsigned long long n_word = (unsigned long long)TX * TY;
    DevBuf small, edges;   // {edge count, its second count} and {largest bin, entries}
    RLC_TRY(small.alloc(32));
    RLC_TRY(cudaMemsetAsync(small.p, 0, 32, s));
    uint32_t* n_edge = small.as<uint32_t>();
    unsigned long long* stats = small.as<unsigned long long>() + 1;
    uint32_t nedges = 0;
    if (ncell > 0) {
        k_edges<<<blocks_for((long long)n_word, 256), 256, 0, s>>>(d_bits, W, H, TX, TY, nullptr, n_edge);
        RLC_TRY(cudaGetLastError());
        RLC_TRY(cudaMemcpyAsync(&nedges, n_edge, sizeof(uint32_t), cudaMemcpyDeviceToHost, s));
        RLC_TRY(cudaStreamSynchronize(s));
    }
    RLC_TRY(edges.alloc((size_t)nedges * sizeof(uint32_t)));
    if (nedges) {
        k_edges<<<blocks_for((long long)n_word, 256), 256, 0, s>>>(d_bits, W, H, TX, TY, edges.as<uint32_t>(), n_edge + 1);
        RLC_TRY(cudaGetLastError());
    }

    // 2. count, scan, fill
    DevBuf counts, start;
    RLC_TRY(counts.alloc(((size_t)nb + 1) * sizeof(uint32_t)));
    RLC_TRY(start.alloc(((size_t)nb + 1) * sizeof(uint32_t)));
    RLC_TRY(cudaMemsetAsync(counts.p, 0, ((size_t)nb + 1) * sizeof(uint32_t), s));
    const long long work = (long long)nedges * nslices;
    // a slice's bins in shared memory where the widest fits a block that leaves room for a second
    uint32_t most = 0;
    for (int a = 0; a < nslices; ++a) most = std::max(most, h_slice_base[a + 1] - h_slice_base[a]);
    const size_t bins_smem = (size_t)most * sizeof(uint32_t);
    const bool by_block = work > 0 && bins_smem <= kProjectSmem && nslices <= 65535;
    const dim3 pgrid((nedges + kProjectChunk - 1) / kProjectChunk, (unsigned)nslices);
    if (by_block) {
        if (bins_smem > 48 * 1024) {   // the limits to the most a table may need: tables are built by several threads
            static std::atomic<unsigned long long> attr0{0}, attr1{0};
            RLC_TRY(ensure_smem_attr(k_project_block<0>, (int)kProjectSmem, attr0));
            RLC_TRY(ensure_smem_attr(k_project_block<1>, (int)kProjectSmem, attr1));
        }
        k_project_block<0><<<pgrid, kProjectThreads, bins_smem, s>>>(g, edges.as<uint32_t>(), nedges, H,
                                                                     counts.as<uint32_t>(), nullptr, nullptr);
        RLC_TRY(cudaGetLastError());
    } else if (work > 0) {
        k_project<0><<<blocks_for(work, 256), 256, 0, s>>>(g, edges.as<uint32_t>(), nedges, H, nslices,
                                                           counts.as<uint32_t>(), nullptr, nullptr);
        RLC_TRY(cudaGetLastError());
    }
    unsigned long long h_stats[2] = {0, 0};
    if (nb > 0) {
        k_count_stats<<<256, 256, 0, s>>>(counts.as<uint32_t>(), nb, stats);
        RLC_TRY(cudaGetLastError());
        RLC_TRY(cudaMemcpyAsync(h_stats, stats, sizeof(h_stats), cudaMemcpyDeviceToHost, s));
        RLC_TRY(cudaStreamSynchronize(s));
    }
    const uint32_t mlen = (uint32_t)h_stats[0];
    if (h_stats[1] >= 0xffffffffull) {   // the CSR offsets are uint32
        snprintf(why, why_len, "CDDT table has %llu entries; the device layout holds < 2^32", h_stats[1]);
        return cudaErrorInvalidValue;
    }
    size_t p2 = 1;
    while (p2 < mlen) p2 <<= 1;
    const size_t smem = p2 * sizeof(float);
    if (smem > kSortSmem) {
        snprintf(why, why_len, "CDDT bin of %u zero points exceeds the in-shared-memory sort (max 51200)", mlen);
        return cudaErrorInvalidValue;
    }
    RLC_TRY(scan_exclusive_u32(counts.as<uint32_t>(), start.as<uint32_t>(), nb, s));
    DevBuf raw;
    RLC_TRY(raw.alloc((size_t)h_stats[1] * sizeof(float)));
    RLC_TRY(cudaMemsetAsync(counts.p, 0, ((size_t)nb + 1) * sizeof(uint32_t), s));
    if (by_block) {
        k_project_block<1><<<pgrid, kProjectThreads, bins_smem, s>>>(g, edges.as<uint32_t>(), nedges, H,
                                                                     counts.as<uint32_t>(), start.as<uint32_t>(),
                                                                     raw.as<float>());
        RLC_TRY(cudaGetLastError());
    } else if (work > 0) {
        k_project<1><<<blocks_for(work, 256), 256, 0, s>>>(g, edges.as<uint32_t>(), nedges, H, nslices,
                                                           counts.as<uint32_t>(), start.as<uint32_t>(),
                                                           raw.as<float>());
        RLC_TRY(cudaGetLastError());
    }

    // 3. sort + unique per bin (counts: the list of long bins)
    DevBuf ucount;
    RLC_TRY(ucount.alloc(((size_t)nb + 1) * sizeof(uint32_t)));
    if (nb > 0) {
        RLC_TRY(cudaMemsetAsync(counts.p, 0, sizeof(uint32_t), s));
        k_sort_bins<<<blocks_for(nb, 8), 256, 0, s>>>(start.as<uint32_t>(), nb, raw.as<float>(), ucount.as<uint32_t>(),
                                                      counts.as<uint32_t>());
        RLC_TRY(cudaGetLastError());
        if (mlen > 256) {
            static std::atomic<unsigned long long> attr{0};
            if (smem > 48 * 1024) RLC_TRY(ensure_smem_attr(k_sort_unique, (int)kSortSmem, attr));
            k_sort_unique<<<2 * 152, 256, smem, s>>>(counts.as<uint32_t>(), start.as<uint32_t>(), raw.as<float>(),
                                                     ucount.as<uint32_t>());
            RLC_TRY(cudaGetLastError());
        }
    }

    // 4. final CSR
    uint32_t* d_bin_start = nullptr;
    float* d_zeros = nullptr;
    RLC_TRY(cudaMalloc(&d_bin_start, ((size_t)nb + 1) * sizeof(uint32_t)));
    cudaError_t e = scan_exclusive_u32(ucount.as<uint32_t>(), d_bin_start, nb, s);
    uint32_t nz = 0;
    if (e == cudaSuccess) e = cudaMemcpy(&nz, d_bin_start + nb, sizeof(uint32_t), cudaMemcpyDeviceToHost);
    if (e == cudaSuccess) e = cudaMalloc(&d_zeros, cddt_zeros_bytes(nz));
    if (e == cudaSuccess && nb > 0) {
        k_copy_bins<<<blocks_for(nb, 8), 256, 0, s>>>(start.as<uint32_t>(), raw.as<float>(), nb, d_bin_start, d_zeros);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    uint32_t* d_slice_base = nullptr;
    if (e == cudaSuccess) e = cudaMalloc(&d_slice_base, (td + 1) * sizeof(uint32_t));
    if (e == cudaSuccess)
        e = cudaMemcpy(d_slice_base, h_slice_base, (td + 1) * sizeof(uint32_t), cudaMemcpyHostToDevice);
    if (e != cudaSuccess) {
        cudaFree(d_bin_start);
        cudaFree(d_zeros);
        cudaFree(d_slice_base);
        return e;
    }
    out->slice_base = d_slice_base;
    out->bin_start = d_bin_start;
    out->zeros = d_zeros;
    out->total_bins = nb;
    out->nzeros = nz;
    return cudaSuccess;
}

void cddt_index_free(CddtIndex* ix) {
    cudaFree(ix->mem);
    *ix = CddtIndex{};
}

cudaError_t cddt_index_build(const CddtBuild& tab, int W, int H, unsigned td, const int* h_widths, const float* h_trans,
                             const float* h_cos, const float* h_sin, const uint32_t* h_slice_base, CddtIndex* ix,
                             cudaStream_t s) {
    cddt_index_free(ix);
    const uint32_t nb = tab.total_bins;
    const unsigned long long nq = 4 * ((unsigned long long)(tab.nzeros >> 2) + 2ull * nb);
    if (nb == 0 || nq + 8 >= (1ull << 32)) return cudaSuccess;
    // slices without zero points (all from td / 2 on, unless a loaded table fills them) have no entries
    std::vector<uint32_t> slice_zero(td + 1);
    DevBuf firsts;
    RLC_TRY(firsts.alloc((td + 1) * sizeof(uint32_t)));
    k_gather_u32<<<blocks_for(td + 1, 256), 256, 0, s>>>(tab.bin_start, tab.slice_base, td + 1, firsts.as<uint32_t>());
    RLC_TRY(cudaGetLastError());
    RLC_TRY(cudaMemcpyAsync(slice_zero.data(), firsts.p, (td + 1) * sizeof(uint32_t), cudaMemcpyDeviceToHost, s));
    RLC_TRY(cudaStreamSynchronize(s));
    std::vector<IndexSlice> sl(td);
    unsigned long long entries = 0;
    for (unsigned a = 0; a < td; ++a) {
        IndexSlice& S = sl[a];
        const float cx = (float)W * h_cos[a], sy = -((float)H * h_sin[a]);
        const float lo = fminf(0.0f, fminf(cx, fminf(sy, cx + sy))), hi = fmaxf(0.0f, fmaxf(cx, fmaxf(sy, cx + sy)));
        const bool used = slice_zero[a + 1] > slice_zero[a] && hi - lo < 1e9f;
        if (slice_zero[a + 1] > slice_zero[a] && !used) return cudaSuccess;
        S = IndexSlice{h_cos[a], h_sin[a], h_trans[a], lo, (uint32_t)h_widths[a], (uint32_t)entries,
                       used ? (uint32_t)((hi - lo) / kCddtBucket) + 2u : 0u, 0u};
        entries += (unsigned long long)h_widths[a] * S.row;
        if (entries >= (1ull << 32)) return cudaSuccess;
    }
    auto up = [](size_t b) { return (b + 255) & ~(size_t)255; };
    const size_t o_q = up(td * sizeof(IndexSlice)), o_i = o_q + up(nq * sizeof(float));
    const size_t o_bad = o_i + up(entries * sizeof(uint32_t)), total = o_bad + 256;
    char* mem = nullptr;
    if (cudaMalloc(&mem, total) != cudaSuccess) {
        cudaGetLastError();
        return cudaSuccess;
    }
    unsigned* bad = reinterpret_cast<unsigned*>(mem + o_bad);
    unsigned h_bad = 0;
    cudaError_t e = cudaMemcpyAsync(mem, sl.data(), td * sizeof(IndexSlice), cudaMemcpyHostToDevice, s);
    if (e == cudaSuccess) e = cudaMemsetAsync(bad, 0, sizeof(unsigned), s);
    if (e == cudaSuccess) {
        k_index_fill<<<blocks_for((long long)nb * 32, 256), 256, 0, s>>>(
            reinterpret_cast<const IndexSlice*>(mem), tab.slice_base, (int)td, nb, tab.bin_start, tab.zeros,
            reinterpret_cast<float*>(mem + o_q), reinterpret_cast<uint32_t*>(mem + o_i), bad);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaMemcpyAsync(&h_bad, bad, sizeof(unsigned), cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    if (e != cudaSuccess || h_bad) {
        cudaFree(mem);
        return e;
    }
    ix->mem = mem;
    ix->slices = reinterpret_cast<const float4*>(mem);
    ix->qz = reinterpret_cast<const float*>(mem + o_q);
    ix->index = reinterpret_cast<const uint32_t*>(mem + o_i);
    return cudaSuccess;
}

cudaError_t cddt_prune(const uint64_t* d_bits, int W, int H, int TY, unsigned td, float max_range,
                       const int* d_widths, const float* d_trans, const float* d_cos, const float* d_sin,
                       CddtBuild* tab, cudaStream_t s) {
    const int nslices = (int)((td + 1) / 2);
    const uint32_t nz = tab->nzeros, nb = tab->total_bins;
    SliceGeom g{d_widths, d_trans, d_cos, d_sin, tab->slice_base};
    DevBuf used, pos;
    RLC_TRY(used.alloc(((size_t)nz + 1) * sizeof(uint32_t)));
    RLC_TRY(pos.alloc(((size_t)nz + 1) * sizeof(uint32_t)));
    RLC_TRY(cudaMemsetAsync(used.p, 0, ((size_t)nz + 1) * sizeof(uint32_t), s));
    const long long ncell = (long long)W * H;
    if (ncell > 0 && nz > 0) {
        DevBuf tag, val, last, need;
        RLC_TRY(tag.alloc((size_t)ncell * sizeof(int)));
        RLC_TRY(val.alloc((size_t)ncell * sizeof(int)));
        RLC_TRY(last.alloc((size_t)ncell * sizeof(int)));
        RLC_TRY(need.alloc(sizeof(unsigned)));
        for (int a = 0; a < nslices; ++a) {
            RLC_TRY(cudaMemsetAsync(need.p, 0, sizeof(unsigned), s));
            k_prune_classify<<<blocks_for(ncell, 256), 256, 0, s>>>(g, a, d_bits, W, H, TY, tab->bin_start,
                                                                    tab->zeros, max_range, used.as<uint32_t>(),
                                                                    tag.as<int>(), val.as<int>(), need.as<unsigned>());
            RLC_TRY(cudaGetLastError());
            unsigned n_need = 0;
            RLC_TRY(cudaMemcpyAsync(&n_need, need.p, sizeof(unsigned), cudaMemcpyDeviceToHost, s));
            RLC_TRY(cudaStreamSynchronize(s));
            if (n_need == 0) continue;
            RLC_TRY((scan_impl<OpMax, true>(tag.as<int>(), last.as<int>(), (size_t)ncell, s)));
            k_prune_stale<<<blocks_for(ncell, 256), 256, 0, s>>>(g, a, W, H, tab->bin_start, tag.as<int>(),
                                                                 last.as<int>(), val.as<int>(), used.as<uint32_t>());
            RLC_TRY(cudaGetLastError());
        }
    }
    // slices >= nslices keep all their entries
    uint32_t first_unpruned = 0;
    {
        uint32_t first_bin = 0;
        std::vector<uint32_t> hsb(td + 1);
        RLC_TRY(cudaMemcpy(hsb.data(), tab->slice_base, (td + 1) * sizeof(uint32_t), cudaMemcpyDeviceToHost));
        first_bin = hsb[nslices];
        RLC_TRY(cudaMemcpy(&first_unpruned, tab->bin_start + first_bin, sizeof(uint32_t), cudaMemcpyDeviceToHost));
    }
    if (nz > 0) {
        k_keep_flags<<<blocks_for(nz, 256), 256, 0, s>>>(used.as<uint32_t>(), first_unpruned, nz);
        RLC_TRY(cudaGetLastError());
    }
    RLC_TRY(scan_exclusive_u32(used.as<uint32_t>(), pos.as<uint32_t>(), nz, s));
    uint32_t nkeep = 0;
    RLC_TRY(cudaMemcpy(&nkeep, pos.as<uint32_t>() + nz, sizeof(uint32_t), cudaMemcpyDeviceToHost));
    float* d_new = nullptr;
    uint32_t* d_new_start = nullptr;
    RLC_TRY(cudaMalloc(&d_new, cddt_zeros_bytes(nkeep)));
    cudaError_t e = cudaMalloc(&d_new_start, ((size_t)nb + 1) * sizeof(uint32_t));
    if (e == cudaSuccess && nz > 0) {
        k_compact_entries<<<blocks_for(nz, 256), 256, 0, s>>>(used.as<uint32_t>(), pos.as<uint32_t>(), nz,
                                                              tab->zeros, d_new);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) {
        k_remap_starts<<<blocks_for((long long)nb + 1, 256), 256, 0, s>>>(tab->bin_start, pos.as<uint32_t>(), nb,
                                                                           d_new_start);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) {
        cudaFree(d_new);
        cudaFree(d_new_start);
        return e;
    }
    cudaFree(tab->zeros);
    cudaFree(tab->bin_start);
    tab->zeros = d_new;
    tab->bin_start = d_new_start;
    tab->nzeros = nkeep;
    return cudaSuccess;
}

}  // namespace rlc
