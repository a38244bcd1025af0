// C ABI (include/rangelibc.h): handle management, host<->device staging,
// argument checking and error reporting around the device kernels.
#include "rangelibc.h"
#include "rlc_internal.cuh"

#include <algorithm>
#include <atomic>
#include <climits>
#include <cmath>
#include <cstdarg>
#include <cstdio>
#include <cstring>
#include <memory>
#include <mutex>
#include <new>
#include <string>
#include <vector>

using namespace rlc;

namespace {

thread_local std::string g_err;

int fail(int code, const char* fmt, ...) {
    char buf[512];
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(buf, sizeof(buf), fmt, ap);
    va_end(ap);
    g_err = buf;
    return code;
}

int cuda_fail(cudaError_t e, const char* what) {
    if (e == cudaErrorMemoryAllocation)
        return fail(RLC_ERR_NOMEM, "%s: %s", what, cudaGetErrorString(e));
    return fail(RLC_ERR_CUDA, "%s: %s", what, cudaGetErrorString(e));
}

#define CUDA_OR_FAIL(expr, what)                       \
    do {                                               \
        cudaError_t _e = (expr);                       \
        if (_e != cudaSuccess) return cuda_fail(_e, what); \
    } while (0)

constexpr double kM2Pi = 6.28318530718;   // RangeLib.h:61
constexpr double kMPi = 3.14159265358979323846;   // M_PI

// float -> int with C truncation, saturating, NaN -> 0 (as the device's cvt.rzi.s32.f32)
inline int host_f2i(float v) {
    if (v != v) return 0;
    if (v >= 2147483648.0f) return INT_MAX;
    if (v <= -2147483904.0f) return INT_MIN;
    return (int)v;
}
constexpr double kEps = 0.00001;          // RangeLib.h:60

}  // namespace

int rlc::set_last_error(int code, const char* msg) {
    g_err = msg ? msg : "";
    return code;
}

// A block of host memory for a map's bits.  Fresh pages that the GPU writes, and their unmapping, cost 12 us
// of a 2048^2 map's 0.6 ms, so the last block of up to kKeep words (1 MB) that a map gave back waits for the
// next one that fits, until the process ends.
struct HostBits {
    static constexpr size_t kKeep = 1u << 17;
    std::unique_ptr<uint64_t[]> p;
    size_t words = 0;

    // at least `n` words, or null; new ones zeroed, so that the GPU writes to pages that are there
    void take(size_t n) {
        Spare& s = spare();
        {
            std::lock_guard<std::mutex> lk(s.mu);
            if (s.words >= n) {
                p = std::move(s.p);
                words = s.words;
                s.words = 0;
            }
        }
        if (!p) {
            p.reset(new (std::nothrow) uint64_t[n]());
            words = n;
        }
    }
    ~HostBits() {
        if (!p || words > kKeep) return;
        Spare& s = spare();
        std::lock_guard<std::mutex> lk(s.mu);
        if (words > s.words) {
            std::swap(p, s.p);
            s.words = words;
        }
    }

private:
    struct Spare {
        std::mutex mu;
        std::unique_ptr<uint64_t[]> p;
        size_t words = 0;
    };
    static Spare& spare() {
        static Spare* s = new Spare;   // (a map may outlive this library's statics)
        return *s;
    }
};

struct rlc_map {
    int device = 0;
    int W = 0, H = 0, TY = 0;
    float world[6] = {1.0f, 0.0f, 0.0f, 0.0f, 0.0f, 1.0f};   // scale, angle, ox, oy, sin, cos
    uint64_t* d_bits = nullptr;
    HostBits h_bits;              // their copy, so that the occupancy can be asked for at any time
    float* d_dt = nullptr;
    float* d_dt_tiled = nullptr;
    uint16_t* d_dt16 = nullptr;
    uint8_t* d_dt8 = nullptr;
    float* d_step = nullptr;
    uint32_t* d_runs = nullptr;   // equal-step runs of the step map (DT_RUNS)
    bool long_runs = true;        // enough of them to be worth reading (ensure_dt)
    std::atomic<int> refs{1};
    std::mutex mu;

    uint8_t* d_free = nullptr;
    void* d_layouts = nullptr;    // one allocation behind every distance-transform layout

    ~rlc_map() {
        cudaFree(d_bits);
        cudaFree(d_layouts);
        cudaFree(d_free);
    }
    // The free distances of Bresenham's walk on first use, a byte per cell.  Where there is no memory for
    // them there are none, and the walk goes cell by cell.  What they add to a map's first Bresenham method:
    // 0.03 ms on 512^2, 0.17 on 2048^2 and 1.5 on 8192^2 with walls, 0.04, 0.25 and 2.7 on empty maps (of
    // which the allocation 0.1 from 4 MB on); a call of 10,000 queries gains 0.03 ms, 4,000 x 61 rays 0.03.
    int ensure_free() {
        std::lock_guard<std::mutex> lk(mu);
        const size_t cells = step_map_cells(W, H);
        if (d_free || cells == 0) return RLC_OK;
        uint8_t* out = nullptr;
        if (cudaMalloc(&out, cells) != cudaSuccess) {
            cudaGetLastError();
            return RLC_OK;
        }
        cudaError_t e = launch_free_map(d_bits, W, H, TY, out, 0);
        if (e == cudaSuccess) e = cudaStreamSynchronize(0);
        if (e != cudaSuccess) {
            cudaFree(out);
            return cuda_fail(e, "free distances");
        }
        d_free = out;
        return RLC_OK;
    }
    // Distance transform and its layouts on first use (RayMarching constructor, RangeLib.h:924).
    // All of them share one allocation (a cudaMalloc + cudaFree pair of 4 MB or more costs ~110 us
    // whatever its size, seven of them cost more than every kernel here), and the searches'
    // scratch is the run map's space, which is written last.
    int ensure_dt() {
        std::lock_guard<std::mutex> lk(mu);
        if (d_dt) return RLC_OK;
        const size_t n = (size_t)W * H, tiled = (size_t)((W + 7) >> 3) * TY * 64;
        size_t total = 0;
        auto room = [&](size_t bytes) {
            const size_t at = total;
            total += (bytes + 255) & ~(size_t)255;
            return at;
        };
        const size_t steps = step_map_cells(W, H);
        const size_t o_dt = room(n * sizeof(float)), o_step = room(steps * sizeof(float));
        const size_t o_tiled = room(tiled * sizeof(float)), o_u16 = room(tiled * sizeof(uint16_t)), o_u8 = room(tiled);
        const size_t o_runs = room(n * sizeof(uint32_t)), o_eq = room(step_eq_words(W, H) * sizeof(uint32_t)), o_share = room(8);
        const size_t sb = edt_scratch_bytes(W, H);
        void* extra = nullptr;   // maps with a side above 16384 need more scratch than the run map holds
        char* base = nullptr;
        cudaError_t e = cudaMalloc(&base, total);
        if (e == cudaSuccess && sb > n * sizeof(uint32_t)) e = cudaMalloc(&extra, sb);
        DtOut o;
        o.dt = (float*)(base + o_dt);
        o.step = steps ? (float*)(base + o_step) : nullptr;
        o.tiled = (float*)(base + o_tiled);
        o.u16 = (uint16_t*)(base + o_u16);
        o.u8 = (uint8_t*)(base + o_u8);
        uint32_t* runs = (uint32_t*)(base + o_runs);
        if (e == cudaSuccess) e = launch_edt(d_bits, W, H, TY, o, extra ? extra : runs, sb, 0);
        unsigned long long share = 0, *d_share = (unsigned long long*)(base + o_share);
        if (e == cudaSuccess && steps && n) e = launch_step_runs(o.step, W, H, (uint32_t*)(base + o_eq), runs, d_share, 0);
        if (e == cudaSuccess && steps && n) e = cudaMemcpyAsync(&share, d_share, sizeof(share), cudaMemcpyDeviceToHost, 0);
        if (e == cudaSuccess) e = cudaStreamSynchronize(0);
        cudaFree(extra);
        if (e != cudaSuccess) {
            cudaFree(base);
            return cuda_fail(e, "distance transform");
        }
        d_layouts = base;
        d_dt = o.dt;
        d_dt_tiled = o.tiled;
        d_dt16 = o.u16;
        d_dt8 = o.u8;
        d_step = o.step;
        d_runs = runs;
        // Runs are long where walls lie along the axes: in a quarter to a half of the free cells of the
        // rectangles-and-disks maps, three quarters of the corridor maps', but 8 % on the reference's
        // basement map, where reading them costs more than it saves (200,000 queries of 300 px from free
        // cells linear / step / runs 42 / 40 / 48 us, 2 M of 500 px 101 / 99 / 105 us).  The line is at a sixth.
        long_runs = 6 * (share & 0xffffffffull) >= share >> 32;
        return RLC_OK;
    }
    void retain() { refs.fetch_add(1); }
    void release() {
        if (refs.fetch_sub(1) == 1) delete this;
    }
};

struct rlc_method {
    rlc_map* map = nullptr;
    int kind = RLC_RM;        // public kind
    int dkind = K_RM;         // device kind
    float mr = 0.0f;
    unsigned td = 0;
    WorldDev world{};
    // CDDT
    std::vector<int> h_widths;
    std::vector<float> h_trans, h_cos, h_sin;
    std::vector<uint32_t> h_slice_base;
    float td_div_2pi = 0.0f, twopi_div_td = 0.0f;
    int* d_widths = nullptr;
    float* d_trans = nullptr;
    float* d_cos = nullptr;
    float* d_sin = nullptr;
    CddtBuild tab;
    CddtIndex index;
    // counts the changes to what a batch's filter table holds of this method: its CDDT table, trig override
    // and sensor model
    unsigned generation = 0;
    // GiantLUTCast
    uint16_t* d_lut = nullptr;
    float max_div_limits = 0.0f, limits_div_max = 0.0f;
    // sensor model
    double* d_table = nullptr;
    int K = 0;
    // staging for host-pointer calls
    void* d_stage = nullptr;
    size_t stage_cap = 0;
    unsigned* d_err = nullptr;
    float* d_trig = nullptr;
    int64_t trig_count = 0;
    // beam-major range bins of the staged fused update (scratch, n x na)
    uint16_t* d_bins = nullptr;
    size_t bins_cap = 0;
    // schedule
    int layout = DT_LINEAR;
    int prefetch = 0;
    int fused_block = 256;
    int tile = 0;             // particles per tile of the fused kernels (0 = auto)
    // No schedule asked for: every call picks its kernels by size (results do not depend on the schedule;
    // rlc_method_get_schedule reports the values above meanwhile).  The fused update has its own word,
    // which autotune changes: it times that call and decides for no other.
    bool pick = true, pick_fused = true;
    bool autotune_pending = false;
    // a schedule of the fused update; pick: what the call chooses by itself
    struct Fused { int layout, block, prefetch, tile; bool pick; };
    // the last autotune: every candidate's schedule and median times (ms) of both stages
    struct TuneResult { Fused f; float first_ms, final_ms; };
    std::vector<TuneResult> tune_results;

    ~rlc_method() {
        cudaFree(d_widths);
        cudaFree(d_trans);
        cudaFree(d_cos);
        cudaFree(d_sin);
        cudaFree(tab.slice_base);
        cudaFree(tab.bin_start);
        cudaFree(tab.zeros);
        cddt_index_free(&index);
        cudaFree(d_table);
        cudaFree(d_stage);
        cudaFree(d_err);
        cudaFree(d_trig);
        cudaFree(d_bins);
        cudaFree(d_lut);
        if (map) map->release();
    }

    // dt_layout: the distance transform's layout that the call reads
    CastParams params(int dt_layout = DT_LINEAR) const {
        CastParams p{};
        p.kind = dkind;
        p.mr = mr;
        p.map.W = map->W;
        p.map.H = map->H;
        p.map.tiles_y = map->TY;
        p.map.dt = dt_layout == DT_TILED ? map->d_dt_tiled : map->d_dt;   // linear for DT_U16 / DT_STAGED
        p.map.dt16 = map->d_dt16;
        p.map.dt8 = map->d_dt8;
        p.map.step = map->d_step;
        p.map.runs = map->d_runs;
        p.map.bits = map->d_bits;
        p.map.free = map->d_free;
        p.cddt.td = td;
        p.cddt.td_div_2pi = td_div_2pi;
        p.cddt.twopi_div_td = twopi_div_td;
        p.cddt.widths = d_widths;
        p.cddt.trans = d_trans;
        p.cddt.cosv = d_cos;
        p.cddt.sinv = d_sin;
        p.cddt.slice_base = tab.slice_base;
        p.glt.lut = d_lut;
        p.glt.td = td;
        p.glt.td_div_2pi = td_div_2pi;
        p.glt.max_div_limits = max_div_limits;
        p.cddt.bin_start = tab.bin_start;
        p.cddt.zeros = tab.zeros;
        p.cddt.slices = index.slices;
        p.cddt.index = index.index;
        p.cddt.qz = index.qz;
        p.world = world;
        p.trig = d_trig;
        p.err = d_err;
        return p;
    }

    // the index of the current CDDT table
    cudaError_t build_index() {
        ++generation;
        return cddt_index_build(tab, map->W, map->H, td, h_widths.data(), h_trans.data(), h_cos.data(), h_sin.data(),
                                h_slice_base.data(), &index, 0);
    }

    int stage(size_t bytes, void** out) {
        if (bytes > stage_cap) {
            cudaFree(d_stage);
            d_stage = nullptr;
            stage_cap = 0;
            size_t cap = bytes + bytes / 4 + 256;
            CUDA_OR_FAIL(cudaMalloc(&d_stage, cap), "staging buffer");
            stage_cap = cap;
        }
        *out = d_stage;
        return RLC_OK;
    }
};

int rlc::method_map_view(const rlc_method* m, MapDev* map, WorldDev* world, float* max_range) {
    if (!m) return fail(RLC_ERR_ARG, "null method handle");
    if (m->dkind != K_RM) return fail(RLC_ERR_ARG, "the learned surrogate is built on a ray-marching method");
    CastParams p = m->params();
    p.map.dt = m->map->d_dt;
    *map = p.map;
    *world = p.world;
    *max_range = m->mr;
    return RLC_OK;
}

namespace {

size_t align256(size_t b) { return (b + 255) & ~(size_t)255; }

WorldDev world_consts(const float* w) {
    WorldDev d;
    d.s = w[0];
    d.inv_s = (float)(1.0 / (double)w[0]);                          // RangeLib.h:442
    d.rc = (float)(-1.0 * (double)w[1] - 3.0 * M_PI / 2.0);         // RangeLib.h:450
    d.ox = w[2];
    d.oy = w[3];
    d.sa = w[4];
    d.ca = w[5];
    return d;
}

// Per-slice constants of CDDTCast (RangeLib.h:1007-1061), host libm.
void cddt_constants(rlc_method* m, const float* cos_tab, const float* sin_tab) {
    const unsigned td = m->td;
    const int W = m->map->W, H = m->map->H;
    m->td_div_2pi = (float)((double)td / kM2Pi);
    m->twopi_div_td = (float)(kM2Pi / (double)(float)td);
    m->h_widths.resize(td);
    m->h_trans.resize(td);
    m->h_cos.resize(td);
    m->h_sin.resize(td);
    m->h_slice_base.resize(td + 1);
    m->h_slice_base[0] = 0;
    // (host code is compiled with -ffp-contract=off: plain IEEE float ops)
    for (unsigned i = 0; i < td; ++i) {
        const float angle = (float)(int)i * m->twopi_div_td;
        const float c = cos_tab ? cos_tab[i] : cosf(angle);
        const float s = sin_tab ? sin_tab[i] : sinf(angle);
        m->h_cos[i] = c;
        m->h_sin[i] = s;
        const float rotated_height = std::fabs((float)W * s) + std::fabs((float)H * c);
        m->h_widths[i] = (int)(unsigned)std::ceil((double)rotated_height - kEps);
        const float left_top = (float)H * c;
        const float right_top = (float)W * s + (float)H * c;
        const float right_bottom = (float)W * s;
        const float inner = (right_bottom < right_top) ? right_bottom : right_top;   // std::min
        const float min_y = (inner < left_top) ? inner : left_top;
        const double tr = -1.0 * (double)min_y - kEps;
        m->h_trans[i] = (float)((0.0 < tr) ? tr : 0.0);                            // std::max(0.0, .)
        m->h_slice_base[i + 1] = m->h_slice_base[i] + (uint32_t)m->h_widths[i];
    }
}

int upload(void** d, const void* h, size_t bytes, const char* what) {
    CUDA_OR_FAIL(cudaMalloc(d, bytes ? bytes : 4), what);
    if (bytes) CUDA_OR_FAIL(cudaMemcpy(*d, h, bytes, cudaMemcpyHostToDevice), what);
    return RLC_OK;
}

int check_method(const rlc_method* m) {
    if (!m) return fail(RLC_ERR_ARG, "null method handle");
    return RLC_OK;
}

// Host buffers of the host-pointer entry points.  Where the GPU can read and
// write pageable host memory coherently (Grace + Blackwell over NVLink-C2C:
// cudaDevAttrPageableMemoryAccess), the kernels run on the caller's buffers
// in place -- no staging copies; elsewhere the buffers are staged through
// device memory with one copy each way.
std::atomic<int> g_host_path{RLC_HOST_AUTO};

bool host_direct() {
    if (g_host_path.load() == RLC_HOST_STAGED) return false;
    static std::atomic<int> cached[64];   // per device: 0 unknown, 1 no, 2 yes
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return false;
    int c = cached[dev].load();
    if (c == 0) {
        int v = 0;
        if (cudaDeviceGetAttribute(&v, cudaDevAttrPageableMemoryAccess, dev) != cudaSuccess) v = 0;
        c = v ? 2 : 1;
        cached[dev].store(c);
    }
    return c == 2;
}

int finish_launch(cudaError_t e, const char* what) {
    if (e != cudaSuccess) return cuda_fail(e, what);
    return RLC_OK;
}

// `layout`, or the linear one where the map is too large for a step map
int map_layout(const rlc_map* map, int layout) {
    return (layout == DT_STEP || layout == DT_RUNS) && !map->d_step ? DT_LINEAR : layout;
}

// layout used by the per-ray kernels (the staged schedule only changes the fused update)
int cast_layout(const rlc_method* m) { return m->layout == DT_STAGED ? DT_LINEAR : map_layout(m->map, m->layout); }

// layout of a cast of `rays` rays.  Without a schedule, ray marching takes the step map, with its
// equal-step runs where the call waits for its longest rays: independent queries (their warps mix
// long and short rays: 2 M queries on 2048^2 linear / step / runs 114 / 110 / 89 us, 200,000 35 / 34 /
// 21, 10,000 19 / 19 / 14, 1,000 on 512^2 9.9 / 9.6 / 10.5), and repeat-angle calls between 16 K and
// 256 K rays (4,000 x 61 23 / 22 / 14 us, 200 x 100 22 / 21 / 12; 1 x 1,081 4.9 / 4.8 / 4.8, 20,000 x
// 1,081 249 / 236 / 256).  The upper line is older than the march that looks for runs at every fourth
// step only: 1,588 x 199 26 / 24 / 18 us and 20,000 x 61 36 / 34 / 31 now lie on its wrong side.
int cast_layout(const rlc_method* m, long long rays, bool independent) {
    if (!m->pick || m->dkind != K_RM) return cast_layout(m);
    if (!m->map->long_runs) return map_layout(m->map, DT_STEP);
    return map_layout(m->map, independent || (rays >= (1ll << 14) && rays < (1ll << 18)) ? DT_RUNS : DT_STEP);
}

// search of a CDDT method's queries (the prefetch schedule) or prefetch of a ray-marching one:
// without a schedule, CDDT queries go by the table's index where it has one
int picked_search(const rlc_method* m) { return m->dkind == K_CDDT && m->index.index ? 3 : 0; }
int cast_search(const rlc_method* m) { return m->pick ? picked_search(m) : m->prefetch; }

// layout of a fused call without a schedule: ray marching takes the step map, with its equal-step
// runs while the call waits for its longest rays and not for its products: 4,000 x 61 step / runs 24 /
// 17 us, 500 x 300 31 / 27, 4,000 x 271 47 / 46, 8,000 x 200 49 / 48; 637 x 849 78 / 80, 4,000 x 1,081
// 117 / 117, 20,000 x 1,081 333 / 342 us.
int picked_fused_layout(const rlc_method* m, int n, int na) {
    if (m->dkind != K_RM) return DT_LINEAR;
    if (!m->map->long_runs) return map_layout(m->map, DT_STEP);
    return map_layout(m->map, (long long)n * na < (2ll << 20) && (na < 512 || n >= 2000) ? DT_RUNS : DT_STEP);
}

int check_trig(const rlc_method* m, long long rays) {
    if (m->d_trig && m->trig_count < rays)
        return fail(RLC_ERR_ARG, "trig override holds %lld rays, call needs %lld", (long long)m->trig_count, rays);
    return RLC_OK;
}

}  // namespace

// ======================================================================= ABI
extern "C" {

int rlc_abi_version(void) { return RLC_ABI_VERSION; }

const char* rlc_last_error(void) { return g_err.c_str(); }

int rlc_device_count(void) {
    int n = 0;
    if (cudaGetDeviceCount(&n) != cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    return n;
}

static int map_create(const uint8_t* occ, int width, int height, bool rows, rlc_map** out) {
    if (!out) return fail(RLC_ERR_ARG, "null output handle");
    *out = nullptr;
    if (width <= 0 || height <= 0) return fail(RLC_ERR_ARG, "map size %dx%d must be positive", width, height);
    if (!occ) return fail(RLC_ERR_ARG, "null occupancy grid");
    if ((long long)width * height > (1ll << 31)) return fail(RLC_ERR_ARG, "map of %dx%d cells is too large", width, height);
    rlc_map* m = new rlc_map();
    cudaGetDevice(&m->device);
    m->W = width;
    m->H = height;
    m->TY = (height + 7) >> 3;
    size_t n = (size_t)width * height;
    size_t words = (size_t)((width + 7) >> 3) * m->TY;
    // the grid is read once: in place where the GPU reads host memory, else staged
    const bool direct = host_direct();
    uint8_t* d_occ = nullptr;
    cudaError_t e = cudaMalloc(&m->d_bits, words * sizeof(uint64_t));
    if (!direct) {
        if (e == cudaSuccess) e = cudaMalloc(&d_occ, n);
        if (e == cudaSuccess) e = cudaMemcpy(d_occ, occ, n, cudaMemcpyHostToDevice);
    }
    if (e == cudaSuccess) e = launch_pack_bits(direct ? occ : d_occ, width, height, rows, m->d_bits, 0);
    m->h_bits.take(words);
    if (e == cudaSuccess && !m->h_bits.p) e = cudaErrorMemoryAllocation;
    if (e == cudaSuccess && direct) {
        e = launch_copy_bits(m->d_bits, words, m->h_bits.p.get(), 0);
        if (e == cudaSuccess) e = cudaStreamSynchronize(0);
    } else if (e == cudaSuccess) {
        e = cudaMemcpy(m->h_bits.p.get(), m->d_bits, words * sizeof(uint64_t), cudaMemcpyDeviceToHost);
    }
    cudaFree(d_occ);
    if (e != cudaSuccess) {
        delete m;
        return cuda_fail(e, "map upload");
    }
    *out = m;
    return RLC_OK;
}

int rlc_map_create(const uint8_t* occ, int width, int height, rlc_map** out) {
    return map_create(occ, width, height, false, out);
}

int rlc_map_create_rows(const uint8_t* rows, int width, int height, rlc_map** out) {
    return map_create(rows, width, height, true, out);
}

int rlc_map_set_world(rlc_map* map, float scale, float angle, float ox, float oy, float sin_angle,
                      float cos_angle) {
    if (!map) return fail(RLC_ERR_ARG, "null map handle");
    map->world[0] = scale;
    map->world[1] = angle;
    map->world[2] = ox;
    map->world[3] = oy;
    map->world[4] = sin_angle;
    map->world[5] = cos_angle;
    return RLC_OK;
}

int rlc_map_destroy(rlc_map* map) {
    if (map) map->release();
    return RLC_OK;
}

int rlc_map_size(const rlc_map* map, int* width, int* height) {
    if (!map) return fail(RLC_ERR_ARG, "null map handle");
    if (width) *width = map->W;
    if (height) *height = map->H;
    return RLC_OK;
}

int rlc_map_occupancy(rlc_map* map, uint8_t* occ_out) {
    if (!map || !occ_out) return fail(RLC_ERR_ARG, "null argument");
    for (int x = 0; x < map->W; ++x) {
        uint8_t* col = occ_out + (size_t)x * map->H;
        const uint64_t* tiles = map->h_bits.p.get() + (size_t)(x >> 3) * map->TY;
        for (int y = 0; y < map->H; y += 8) {
            // the tile's eight cells of this column, a byte each: the product puts bit k at bit 8 k (k < 7)
            const uint64_t b = (tiles[y >> 3] >> ((x & 7) << 3)) & 0xFFu;
            const uint64_t cells = (((b & 0x7Fu) * 0x40810204081ull) & 0x0101010101010101ull) | (b >> 7) << 56;
            if (y + 8 <= map->H) std::memcpy(col + y, &cells, 8);
            else
                for (int k = 0; y + k < map->H; ++k) col[y + k] = (uint8_t)(cells >> (8 * k));
        }
    }
    return RLC_OK;
}

int rlc_map_distance_transform(rlc_map* map, float* dt_out) {
    if (!map || !dt_out) return fail(RLC_ERR_ARG, "null argument");
    int rc = map->ensure_dt();
    if (rc) return rc;
    CUDA_OR_FAIL(cudaMemcpy(dt_out, map->d_dt, (size_t)map->W * map->H * sizeof(float), cudaMemcpyDeviceToHost),
                 "distance transform export");
    return RLC_OK;
}

int rlc_map_edge_map(rlc_map* map, uint8_t* edge_out) {
    if (!map || !edge_out) return fail(RLC_ERR_ARG, "null argument");
    size_t n = (size_t)map->W * map->H;
    uint8_t* d = nullptr;
    CUDA_OR_FAIL(cudaMalloc(&d, n), "edge map");
    cudaError_t e = launch_edge_map(map->d_bits, map->W, map->H, map->TY, d, 0);
    if (e == cudaSuccess) e = cudaMemcpy(edge_out, d, n, cudaMemcpyDeviceToHost);
    cudaFree(d);
    return finish_launch(e, "edge map");
}

// GiantLUTCast constructor (RangeLib.h:1782-1818; cached constants, 16-bit entries): the
// angles i * M_2PI_div_theta_discretization, their host-libm cosf/sinf, and one ray march
// per (cell corner, angle) on the device
static int glt_build(rlc_method* m, const float* cos_tab, const float* sin_tab) {
    cddt_constants(m, cos_tab, sin_tab);   // td_div_2pi, twopi_div_td and the per-angle cos/sin
    m->max_div_limits = m->mr / 65535;
    m->limits_div_max = 65535 / m->mr;
    const size_t cells = (size_t)m->map->W * m->map->H;
    int rc = upload((void**)&m->d_cos, m->h_cos.data(), m->td * sizeof(float), "GLT cos");
    if (!rc) rc = upload((void**)&m->d_sin, m->h_sin.data(), m->td * sizeof(float), "GLT sin");
    if (rc) return rc;
    cudaError_t e = cudaMalloc(&m->d_lut, (cells * m->td > 0 ? cells * m->td : 1) * sizeof(uint16_t));
    if (e != cudaSuccess) {
        m->d_lut = nullptr;
        return fail(RLC_ERR_NOMEM, "GiantLUTCast table of %zu bytes: %s", cells * m->td * sizeof(uint16_t),
                    cudaGetErrorString(e));
    }
    CastParams p = m->params();
    p.map.dt = m->map->d_dt;
    e = launch_glt_build(p.map, m->mr, m->td, m->d_cos, m->d_sin, m->limits_div_max, m->d_lut, 0);
    if (e == cudaSuccess) e = cudaStreamSynchronize(0);
    return e == cudaSuccess ? RLC_OK : cuda_fail(e, "GiantLUTCast construction");
}

static int method_create(rlc_map* map, int kind, float max_range, unsigned td, const float* cos_tab,
                         const float* sin_tab, rlc_method** out) {
    if (!out) return fail(RLC_ERR_ARG, "null output handle");
    *out = nullptr;
    if (!map) return fail(RLC_ERR_ARG, "null map handle");
    if (kind < RLC_BL || kind > RLC_GLT) return fail(RLC_ERR_ARG, "unknown method kind %d", kind);
    if (!std::isfinite(max_range)) return fail(RLC_ERR_ARG, "max_range must be finite");
    bool cddt = kind == RLC_CDDT || kind == RLC_PCDDT;
    const bool glt = kind == RLC_GLT;
    if (cddt && td < 2) return fail(RLC_ERR_ARG, "theta_discretization %u must be >= 2", td);
    if (glt && td < 1) return fail(RLC_ERR_ARG, "theta_discretization must be >= 1");
    if (glt && !(max_range > 0.0f)) return fail(RLC_ERR_ARG, "GiantLUTCast needs max_range > 0");
    rlc_method* m = new rlc_method();
    map->retain();
    m->map = map;
    m->kind = kind;
    m->dkind = kind == RLC_BL ? K_BL : (cddt ? K_CDDT : (glt ? K_GLT : K_RM));
    m->mr = max_range;
    m->td = (cddt || glt) ? td : 0;
    m->world = world_consts(map->world);
    int rc = RLC_OK;
    cudaError_t e = cudaMalloc(&m->d_err, sizeof(unsigned));
    if (e == cudaSuccess) e = cudaMemset(m->d_err, 0, sizeof(unsigned));
    if (e != cudaSuccess) rc = cuda_fail(e, "method state");
    if (!rc && (m->dkind == K_RM || glt)) rc = map->ensure_dt();
    if (!rc && m->dkind == K_BL) rc = map->ensure_free();
    if (!rc && glt) rc = glt_build(m, cos_tab, sin_tab);
    if (!rc && cddt) {
        cddt_constants(m, cos_tab, sin_tab);
        rc = upload((void**)&m->d_widths, m->h_widths.data(), td * sizeof(int), "cddt widths");
        if (!rc) rc = upload((void**)&m->d_trans, m->h_trans.data(), td * sizeof(float), "cddt translations");
        if (!rc) rc = upload((void**)&m->d_cos, m->h_cos.data(), td * sizeof(float), "cddt cos");
        if (!rc) rc = upload((void**)&m->d_sin, m->h_sin.data(), td * sizeof(float), "cddt sin");
        if (!rc) {
            char why[256] = {0};
            e = cddt_build(map->d_bits, map->W, map->H, map->TY, td, m->d_widths, m->d_trans, m->d_cos, m->d_sin,
                           m->h_slice_base.data(), &m->tab, 0, why, sizeof(why));
            if (e != cudaSuccess) rc = why[0] ? fail(RLC_ERR_ARG, "%s", why) : cuda_fail(e, "CDDT construction");
        }
        if (!rc && kind == RLC_PCDDT) {
            e = cddt_prune(map->d_bits, map->W, map->H, map->TY, td, max_range, m->d_widths, m->d_trans, m->d_cos,
                           m->d_sin, &m->tab, 0);
            if (e != cudaSuccess) rc = cuda_fail(e, "CDDT prune");
        }
        if (!rc && (e = m->build_index()) != cudaSuccess) rc = cuda_fail(e, "CDDT index");
    }
    if (rc) {
        delete m;
        return rc;
    }
    *out = m;
    return RLC_OK;
}

int rlc_method_create(rlc_map* map, int kind, float max_range, unsigned theta_disc, rlc_method** out) {
    return method_create(map, kind, max_range, theta_disc, nullptr, nullptr, out);
}

int rlc_method_create_cddt_trig(rlc_map* map, int kind, float max_range, unsigned theta_disc,
                                const float* cos_tab, const float* sin_tab, rlc_method** out) {
    if (kind != RLC_CDDT && kind != RLC_PCDDT && kind != RLC_GLT)
        return fail(RLC_ERR_ARG, "trig tables apply to CDDT and GLT kinds");
    if (!cos_tab || !sin_tab) return fail(RLC_ERR_ARG, "null trig table");
    return method_create(map, kind, max_range, theta_disc, cos_tab, sin_tab, out);
}

int rlc_method_destroy(rlc_method* m) {
    delete m;
    return RLC_OK;
}

int rlc_method_info(const rlc_method* m, int* kind, float* max_range, unsigned* theta_disc) {
    if (int rc = check_method(m)) return rc;
    if (kind) *kind = m->kind;
    if (max_range) *max_range = m->mr;
    if (theta_disc) *theta_disc = m->td;
    return RLC_OK;
}

int rlc_method_device_flags(rlc_method* m, unsigned* flags) {
    if (int rc = check_method(m)) return rc;
    unsigned f = 0;
    CUDA_OR_FAIL(cudaDeviceSynchronize(), "device flags");
    CUDA_OR_FAIL(cudaMemcpy(&f, m->d_err, sizeof(unsigned), cudaMemcpyDeviceToHost), "device flags");
    CUDA_OR_FAIL(cudaMemset(m->d_err, 0, sizeof(unsigned)), "device flags");
    if (flags) *flags = f;
    return RLC_OK;
}

int rlc_cddt_prune(rlc_method* m, float max_range) {
    if (int rc = check_method(m)) return rc;
    if (m->dkind != K_CDDT) return fail(RLC_ERR_STATE, "prune applies to CDDT methods");
    cudaError_t e = cddt_prune(m->map->d_bits, m->map->W, m->map->H, m->map->TY, m->td, max_range, m->d_widths,
                               m->d_trans, m->d_cos, m->d_sin, &m->tab, 0);
    if (e == cudaSuccess) e = m->build_index();
    return finish_launch(e, "CDDT prune");
}

int rlc_cddt_table_size(rlc_method* m, int64_t* num_bins, int64_t* num_zeros) {
    if (int rc = check_method(m)) return rc;
    if (m->dkind != K_CDDT) return fail(RLC_ERR_STATE, "not a CDDT method");
    if (num_bins) *num_bins = m->tab.total_bins;
    if (num_zeros) *num_zeros = m->tab.nzeros;
    return RLC_OK;
}

int rlc_cddt_table_export(rlc_method* m, int* widths, float* trans, int64_t* bin_len, float* zeros) {
    if (int rc = check_method(m)) return rc;
    if (m->dkind != K_CDDT) return fail(RLC_ERR_STATE, "not a CDDT method");
    if (widths) std::memcpy(widths, m->h_widths.data(), m->td * sizeof(int));
    if (trans) std::memcpy(trans, m->h_trans.data(), m->td * sizeof(float));
    if (bin_len) {
        std::vector<uint32_t> st(m->tab.total_bins + 1);
        CUDA_OR_FAIL(cudaMemcpy(st.data(), m->tab.bin_start, st.size() * sizeof(uint32_t), cudaMemcpyDeviceToHost),
                     "CDDT export");
        for (uint32_t b = 0; b < m->tab.total_bins; ++b) bin_len[b] = (int64_t)st[b + 1] - st[b];
    }
    if (zeros && m->tab.nzeros)
        CUDA_OR_FAIL(cudaMemcpy(zeros, m->tab.zeros, (size_t)m->tab.nzeros * sizeof(float), cudaMemcpyDeviceToHost),
                     "CDDT export");
    return RLC_OK;
}

int rlc_cddt_table_load(rlc_method* m, const float* trans, const int64_t* bin_len, const float* zeros,
                        int64_t num_zeros) {
    if (int rc = check_method(m)) return rc;
    if (m->dkind != K_CDDT) return fail(RLC_ERR_STATE, "not a CDDT method");
    if (!trans || !bin_len || (num_zeros > 0 && !zeros)) return fail(RLC_ERR_ARG, "null table argument");
    if (num_zeros < 0 || num_zeros >= (int64_t)0xffffffffll) return fail(RLC_ERR_ARG, "bad zero count");
    const uint32_t nb = m->tab.total_bins;
    std::vector<uint32_t> st(nb + 1);
    st[0] = 0;
    for (uint32_t b = 0; b < nb; ++b) {
        if (bin_len[b] < 0) return fail(RLC_ERR_ARG, "negative bin length");
        uint64_t next = (uint64_t)st[b] + (uint64_t)bin_len[b];
        if (next > (uint64_t)num_zeros) return fail(RLC_ERR_ARG, "bin lengths exceed num_zeros");
        st[b + 1] = (uint32_t)next;
    }
    if (st[nb] != (uint32_t)num_zeros) return fail(RLC_ERR_ARG, "bin lengths sum to %u, not %lld", st[nb], (long long)num_zeros);
    uint32_t* d_st = nullptr;
    float* d_z = nullptr;
    if (int rc = upload((void**)&d_st, st.data(), st.size() * sizeof(uint32_t), "CDDT load")) return rc;
    cudaError_t ez = cudaMalloc((void**)&d_z, cddt_zeros_bytes((size_t)num_zeros));
    if (ez == cudaSuccess && num_zeros)
        ez = cudaMemcpy(d_z, zeros, (size_t)num_zeros * sizeof(float), cudaMemcpyHostToDevice);
    if (ez != cudaSuccess) {
        cudaFree(d_st);
        cudaFree(d_z);
        return cuda_fail(ez, "CDDT load");
    }
    cudaFree(m->tab.bin_start);
    cudaFree(m->tab.zeros);
    m->tab.bin_start = d_st;
    m->tab.zeros = d_z;
    m->tab.nzeros = (uint32_t)num_zeros;
    std::memcpy(m->h_trans.data(), trans, m->td * sizeof(float));
    CUDA_OR_FAIL(cudaMemcpy(m->d_trans, trans, m->td * sizeof(float), cudaMemcpyHostToDevice), "CDDT load");
    CUDA_OR_FAIL(m->build_index(), "CDDT load");
    return RLC_OK;
}

int rlc_method_set_trig_override(rlc_method* m, const float* trig, int64_t count) {
    if (int rc = check_method(m)) return rc;
    ++m->generation;
    cudaFree(m->d_trig);
    m->d_trig = nullptr;
    m->trig_count = 0;
    if (!trig || count <= 0) return RLC_OK;
    if (int rc = upload((void**)&m->d_trig, trig, (size_t)count * 2 * sizeof(float), "trig override")) return rc;
    m->trig_count = count;
    return RLC_OK;
}

int rlc_set_host_path(int mode) {
    if (mode != RLC_HOST_AUTO && mode != RLC_HOST_STAGED) return fail(RLC_ERR_ARG, "host path mode %d", mode);
    g_host_path.store(mode);
    return RLC_OK;
}

int rlc_host_path(int* direct) {
    if (!direct) return fail(RLC_ERR_ARG, "null output");
    *direct = host_direct() ? 1 : 0;
    return RLC_OK;
}

int rlc_glt_table(rlc_method* m, uint16_t* lut_out) {
    if (int rc = check_method(m)) return rc;
    if (m->dkind != K_GLT) return fail(RLC_ERR_STATE, "not a GiantLUTCast method");
    if (!lut_out) return fail(RLC_ERR_ARG, "null output");
    const size_t n = (size_t)m->map->W * m->map->H * m->td;
    if (n) CUDA_OR_FAIL(cudaMemcpy(lut_out, m->d_lut, n * sizeof(uint16_t), cudaMemcpyDeviceToHost), "GLT export");
    return RLC_OK;
}

int rlc_cddt_calc_range_pair(rlc_method* m, float x, float y, float heading, float* r, float* r_inv) {
    if (int rc = check_method(m)) return rc;
    if (m->dkind != K_CDDT) return fail(RLC_ERR_STATE, "calc_range_pair applies to CDDT methods");
    if (!r || !r_inv) return fail(RLC_ERR_ARG, "null output");
    void* st = nullptr;
    if (int rc = m->stage(2 * sizeof(float), &st)) return rc;
    CastParams p = m->params();
    CUDA_OR_FAIL(launch_cddt_pair(p, x, y, heading, (float*)st, 0), "calc_range_pair");
    float h[2];
    CUDA_OR_FAIL(cudaMemcpy(h, st, sizeof(h), cudaMemcpyDeviceToHost), "calc_range_pair");
    *r = h[0];
    *r_inv = h[1];
    return RLC_OK;
}

// the loop constants of calc_range_many_radial_optimized (RangeLib.h:636-646) and the
// heading offset of each loop index, accumulated as the reference does (angle += step)
static void radial_plan(int num_rays, float min_angle, float max_angle, int* mp, int* off, std::vector<float>* ang) {
    const float step = (max_angle - min_angle) / (float)(num_rays - 1);
    *mp = (int)((double)(float)num_rays / 3.0);
    const float off_f = (float)(((double)num_rays - 1.0) * kMPi / (double)(max_angle - min_angle));
    *off = host_f2i(std::round(off_f));
    const int A = std::max(*mp + 1, *off);
    ang->resize(A > 0 ? A : 1);
    float angle = min_angle;
    for (int a = 0; a < A; ++a) {
        (*ang)[a] = angle;
        angle += step;
    }
}

int rlc_cddt_calc_range_many_radial(rlc_method* m, const float* ins, float* outs, int n, int num_rays,
                                    float min_angle, float max_angle, unsigned flags, void* stream) {
    if (int rc = check_method(m)) return rc;
    if (m->dkind != K_CDDT) return fail(RLC_ERR_STATE, "calc_range_many_radial_optimized applies to CDDT methods");
    if (n < 0 || num_rays < 0) return fail(RLC_ERR_ARG, "negative size");
    if ((long long)n * num_rays == 0) return RLC_OK;
    if (!ins || !outs) return fail(RLC_ERR_ARG, "null array");
    int mp = 0, off = 0;
    std::vector<float> ang;
    radial_plan(num_rays, min_angle, max_angle, &mp, &off, &ang);
    if ((long long)ang.size() > (1ll << 24)) return fail(RLC_ERR_ARG, "beam offset %d out of range", off);
    cudaStream_t s = (cudaStream_t)stream;
    CastParams p = m->params();
    const size_t b_ang = align256(ang.size() * sizeof(float));
    const size_t b_in = (flags & RLC_DEVICE_PTRS) ? 0 : align256((size_t)n * 3 * sizeof(float));
    const size_t b_out = (flags & RLC_DEVICE_PTRS) ? 0 : (size_t)n * num_rays * sizeof(float);
    void* st = nullptr;
    if (int rc = m->stage(b_ang + b_in + b_out, &st)) return rc;
    float* d_ang = (float*)st;
    CUDA_OR_FAIL(cudaMemcpyAsync(d_ang, ang.data(), ang.size() * sizeof(float), cudaMemcpyHostToDevice, s), "H2D");
    if (flags & RLC_DEVICE_PTRS)
        return finish_launch(launch_cddt_radial(p, ins, d_ang, outs, n, num_rays, mp, off, s), "radial");
    if (host_direct()) {
        CUDA_OR_FAIL(launch_cddt_radial(p, ins, d_ang, outs, n, num_rays, mp, off, s), "radial");
        CUDA_OR_FAIL(cudaStreamSynchronize(s), "radial");
        return RLC_OK;
    }
    float* d_in = (float*)((char*)st + b_ang);
    float* d_out = (float*)((char*)st + b_ang + b_in);
    CUDA_OR_FAIL(cudaMemcpyAsync(d_in, ins, (size_t)n * 3 * sizeof(float), cudaMemcpyHostToDevice, s), "H2D");
    // positions the reference does not write keep the caller's values
    CUDA_OR_FAIL(cudaMemcpyAsync(d_out, outs, b_out, cudaMemcpyHostToDevice, s), "H2D");
    CUDA_OR_FAIL(launch_cddt_radial(p, d_in, d_ang, d_out, n, num_rays, mp, off, s), "radial");
    CUDA_OR_FAIL(cudaMemcpyAsync(outs, d_out, b_out, cudaMemcpyDeviceToHost, s), "D2H");
    CUDA_OR_FAIL(cudaStreamSynchronize(s), "radial");
    return RLC_OK;
}

int rlc_calc_range(rlc_method* m, float x, float y, float heading, float* out) {
    if (int rc = check_method(m)) return rc;
    if (!out) return fail(RLC_ERR_ARG, "null output");
    float in[3] = {x, y, heading};
    return rlc_calc_range_many(m, in, out, 1, RLC_NO_WORLD, nullptr);
}

int rlc_calc_range_many(rlc_method* m, const float* ins, float* outs, int n, unsigned flags, void* stream) {
    if (int rc = check_method(m)) return rc;
    if (n < 0) return fail(RLC_ERR_ARG, "negative query count");
    if (n == 0) return RLC_OK;
    if (!ins || !outs) return fail(RLC_ERR_ARG, "null array");
    if (int rc = check_trig(m, n)) return rc;
    cudaStream_t s = (cudaStream_t)stream;
    const int layout = cast_layout(m, n, true);
    CastParams p = m->params(layout);
    bool world = !(flags & RLC_NO_WORLD);
    if (flags & RLC_DEVICE_PTRS)
        return finish_launch(launch_calc_range_many(p, layout, cast_search(m), world, ins, outs, n, s), "calc_range_many");
    if (host_direct()) {
        CUDA_OR_FAIL(launch_calc_range_many(p, layout, cast_search(m), world, ins, outs, n, s), "calc_range_many");
        CUDA_OR_FAIL(cudaStreamSynchronize(s), "calc_range_many");
        return RLC_OK;
    }
    size_t bin = align256((size_t)n * 3 * sizeof(float));
    void* st = nullptr;
    if (int rc = m->stage(bin + (size_t)n * sizeof(float), &st)) return rc;
    float* d_in = (float*)st;
    float* d_out = (float*)((char*)st + bin);
    CUDA_OR_FAIL(cudaMemcpyAsync(d_in, ins, (size_t)n * 3 * sizeof(float), cudaMemcpyHostToDevice, s), "H2D");
    CUDA_OR_FAIL(launch_calc_range_many(p, layout, cast_search(m), world, d_in, d_out, n, s), "calc_range_many");
    CUDA_OR_FAIL(cudaMemcpyAsync(outs, d_out, (size_t)n * sizeof(float), cudaMemcpyDeviceToHost, s), "D2H");
    CUDA_OR_FAIL(cudaStreamSynchronize(s), "calc_range_many");
    return RLC_OK;
}

int rlc_calc_range_repeat_angles(rlc_method* m, const float* ins, const float* angles, float* outs, int n, int na,
                                 unsigned flags, void* stream) {
    if (int rc = check_method(m)) return rc;
    if (n < 0 || na < 0) return fail(RLC_ERR_ARG, "negative size");
    if ((long long)n * na == 0) return RLC_OK;
    if ((long long)n * na > (1ll << 31) - 1) return fail(RLC_ERR_ARG, "too many rays in one call");
    if (!ins || !angles || !outs) return fail(RLC_ERR_ARG, "null array");
    if (int rc = check_trig(m, (long long)n * na)) return rc;
    cudaStream_t s = (cudaStream_t)stream;
    const int layout = cast_layout(m, (long long)n * na, false);
    CastParams p = m->params(layout);
    if (flags & RLC_DEVICE_PTRS)
        return finish_launch(launch_repeat_angles(p, layout, cast_search(m), ins, angles, outs, n, na, s), "repeat_angles");
    if (host_direct()) {
        CUDA_OR_FAIL(launch_repeat_angles(p, layout, cast_search(m), ins, angles, outs, n, na, s), "repeat_angles");
        CUDA_OR_FAIL(cudaStreamSynchronize(s), "repeat_angles");
        return RLC_OK;
    }
    size_t b0 = align256((size_t)n * 3 * sizeof(float));
    size_t b1 = align256((size_t)na * sizeof(float));
    void* st = nullptr;
    if (int rc = m->stage(b0 + b1 + (size_t)n * na * sizeof(float), &st)) return rc;
    float* d_in = (float*)st;
    float* d_ang = (float*)((char*)st + b0);
    float* d_out = (float*)((char*)st + b0 + b1);
    CUDA_OR_FAIL(cudaMemcpyAsync(d_in, ins, (size_t)n * 3 * sizeof(float), cudaMemcpyHostToDevice, s), "H2D");
    CUDA_OR_FAIL(cudaMemcpyAsync(d_ang, angles, (size_t)na * sizeof(float), cudaMemcpyHostToDevice, s), "H2D");
    CUDA_OR_FAIL(launch_repeat_angles(p, layout, cast_search(m), d_in, d_ang, d_out, n, na, s), "repeat_angles");
    CUDA_OR_FAIL(cudaMemcpyAsync(outs, d_out, (size_t)n * na * sizeof(float), cudaMemcpyDeviceToHost, s), "D2H");
    CUDA_OR_FAIL(cudaStreamSynchronize(s), "repeat_angles");
    return RLC_OK;
}

int rlc_set_sensor_model(rlc_method* m, const double* table, int K) {
    if (int rc = check_method(m)) return rc;
    if (!table || K <= 0) return fail(RLC_ERR_ARG, "sensor model needs a K x K table with K > 0");
    if ((long long)K * K > (1ll << 28)) return fail(RLC_ERR_ARG, "sensor table too large");
    ++m->generation;
    cudaFree(m->d_table);
    m->d_table = nullptr;
    m->K = 0;
    if (int rc = upload((void**)&m->d_table, table, (size_t)K * K * sizeof(double), "sensor model")) {
        cudaFree(m->d_table);
        m->d_table = nullptr;
        return rc;
    }
    m->K = K;
    return RLC_OK;
}

int rlc_eval_sensor_model(rlc_method* m, const float* obs, const float* ranges, double* outs, int na, int n,
                          unsigned flags, void* stream) {
    if (int rc = check_method(m)) return rc;
    if (!m->d_table) return fail(RLC_ERR_STATE, "set_sensor_model has not been called");
    if (n < 0 || na < 0) return fail(RLC_ERR_ARG, "negative size");
    if (n == 0) return RLC_OK;
    if (!outs || (na > 0 && (!obs || !ranges))) return fail(RLC_ERR_ARG, "null array");
    if (na > 16384) return fail(RLC_ERR_ARG, "at most 16384 rays per particle");
    cudaStream_t s = (cudaStream_t)stream;
    CastParams p = m->params();
    SensorDev sm{m->d_table, m->K};
    if (flags & RLC_DEVICE_PTRS)
        return finish_launch(launch_eval_sensor(p, sm, obs, ranges, outs, na, n, s), "eval_sensor_model");
    if (host_direct()) {
        CUDA_OR_FAIL(launch_eval_sensor(p, sm, obs, ranges, outs, na, n, s), "eval_sensor_model");
        CUDA_OR_FAIL(cudaStreamSynchronize(s), "eval_sensor_model");
        return RLC_OK;
    }
    size_t b0 = align256((size_t)na * sizeof(float));
    size_t b1 = align256((size_t)n * na * sizeof(float));
    void* st = nullptr;
    if (int rc = m->stage(b0 + b1 + (size_t)n * sizeof(double), &st)) return rc;
    float* d_obs = (float*)st;
    float* d_rng = (float*)((char*)st + b0);
    double* d_out = (double*)((char*)st + b0 + b1);
    if (na) {
        CUDA_OR_FAIL(cudaMemcpyAsync(d_obs, obs, (size_t)na * sizeof(float), cudaMemcpyHostToDevice, s), "H2D");
        CUDA_OR_FAIL(cudaMemcpyAsync(d_rng, ranges, (size_t)n * na * sizeof(float), cudaMemcpyHostToDevice, s), "H2D");
    }
    CUDA_OR_FAIL(launch_eval_sensor(p, sm, d_obs, d_rng, d_out, na, n, s), "eval_sensor_model");
    CUDA_OR_FAIL(cudaMemcpyAsync(outs, d_out, (size_t)n * sizeof(double), cudaMemcpyDeviceToHost, s), "D2H");
    CUDA_OR_FAIL(cudaStreamSynchronize(s), "eval_sensor_model");
    return RLC_OK;
}

static int fused_device(rlc_method* m, const float* ins, const float* angles, const float* obs, double* w, int n,
                        int na, cudaStream_t s);

int rlc_calc_range_repeat_angles_eval_sensor_model(rlc_method* m, const float* ins, const float* angles,
                                                   const float* obs, double* weights, int n, int na,
                                                   unsigned flags, void* stream) {
    if (int rc = check_method(m)) return rc;
    if (!m->d_table) return fail(RLC_ERR_STATE, "set_sensor_model has not been called");
    if (n < 0 || na < 0) return fail(RLC_ERR_ARG, "negative size");
    if (n == 0) return RLC_OK;
    if (!ins || !weights || (na > 0 && (!angles || !obs))) return fail(RLC_ERR_ARG, "null array");
    if (na > 16384) return fail(RLC_ERR_ARG, "at most 16384 beams per particle");
    if ((long long)n * na > (1ll << 31) - 1) return fail(RLC_ERR_ARG, "too many rays in one call");
    if (int rc = check_trig(m, (long long)n * na)) return rc;
    cudaStream_t s = (cudaStream_t)stream;
    if (flags & RLC_DEVICE_PTRS) return fused_device(m, ins, angles, obs, weights, n, na, s);
    if (host_direct()) {
        if (int rc = fused_device(m, ins, angles, obs, weights, n, na, s)) return rc;
        CUDA_OR_FAIL(cudaStreamSynchronize(s), "fused sensor model");
        return RLC_OK;
    }
    size_t b0 = align256((size_t)n * 3 * sizeof(float));
    size_t b1 = align256((size_t)na * sizeof(float));
    size_t b2 = align256((size_t)na * sizeof(float));
    void* st = nullptr;
    if (int rc = m->stage(b0 + b1 + b2 + (size_t)n * sizeof(double), &st)) return rc;
    float* d_in = (float*)st;
    float* d_ang = (float*)((char*)st + b0);
    float* d_obs = (float*)((char*)st + b0 + b1);
    double* d_w = (double*)((char*)st + b0 + b1 + b2);
    CUDA_OR_FAIL(cudaMemcpyAsync(d_in, ins, (size_t)n * 3 * sizeof(float), cudaMemcpyHostToDevice, s), "H2D");
    if (na) {
        CUDA_OR_FAIL(cudaMemcpyAsync(d_ang, angles, (size_t)na * sizeof(float), cudaMemcpyHostToDevice, s), "H2D");
        CUDA_OR_FAIL(cudaMemcpyAsync(d_obs, obs, (size_t)na * sizeof(float), cudaMemcpyHostToDevice, s), "H2D");
    }
    if (int rc = fused_device(m, d_in, d_ang, d_obs, d_w, n, na, s)) return rc;
    CUDA_OR_FAIL(cudaMemcpyAsync(weights, d_w, (size_t)n * sizeof(double), cudaMemcpyDeviceToHost, s), "D2H");
    CUDA_OR_FAIL(cudaStreamSynchronize(s), "fused sensor model");
    return RLC_OK;
}

static int ensure_bins(rlc_method* m, size_t count) {
    if (count <= m->bins_cap) return RLC_OK;
    cudaFree(m->d_bins);
    m->d_bins = nullptr;
    m->bins_cap = 0;
    CUDA_OR_FAIL(cudaMalloc(&m->d_bins, count * sizeof(uint16_t)), "staged update scratch");
    m->bins_cap = count;
    return RLC_OK;
}

// the fused update under one schedule (ensure_bins first for DT_STAGED)
static cudaError_t launch_fused_as(const rlc_method* m, const rlc_method::Fused& f, const float* ins, const float* angles,
                                   const float* obs, double* w, int n, int na, cudaStream_t s) {
    const SensorDev sm{m->d_table, m->K};
    if (f.pick) {
        const int layout = picked_fused_layout(m, n, na);
        return launch_fused(m->params(layout), layout, picked_search(m), sm, ins, angles, obs, w, n, na, 0, 0, true, s);
    }
    if (f.layout == DT_STAGED && m->dkind == K_RM)
        return launch_fused_staged(m->params(), sm, ins, angles, obs, w, n, na, f.tile, m->d_bins, s);
    const int layout = f.layout == DT_STAGED ? DT_LINEAR : map_layout(m->map, f.layout);
    return launch_fused(m->params(layout), layout, f.prefetch, sm, ins, angles, obs, w, n, na, f.block, f.tile, false, s);
}

static int fused_device(rlc_method* m, const float* ins, const float* angles, const float* obs, double* w, int n,
                        int na, cudaStream_t s) {
    if (m->autotune_pending) {
        m->autotune_pending = false;
        int rc = rlc_method_autotune(m, ins, angles, obs, w, n, na, s);
        if (rc) return rc;
    }
    const rlc_method::Fused f{m->layout, m->fused_block, m->prefetch, m->tile, m->pick_fused};
    if (!f.pick && f.layout == DT_STAGED && m->dkind == K_RM)
        if (int rc = ensure_bins(m, (size_t)n * na)) return rc;
    return finish_launch(launch_fused_as(m, f, ins, angles, obs, w, n, na, s), "fused sensor model");
}

int rlc_trig_eval(const float* x, float* sincos, int64_t n, unsigned flags, void* stream) {
    if (n < 0) return fail(RLC_ERR_ARG, "negative size");
    if (n == 0) return RLC_OK;
    if (!x || !sincos) return fail(RLC_ERR_ARG, "null array");
    if (flags & RLC_DEVICE_PTRS) {
        CUDA_OR_FAIL(launch_trig_eval(x, sincos, (long long)n, (cudaStream_t)stream), "trig eval");
        return RLC_OK;
    }
    float* d = nullptr;
    const size_t bx = align256((size_t)n * sizeof(float));
    CUDA_OR_FAIL(cudaMalloc(&d, bx + (size_t)n * 2 * sizeof(float)), "trig eval allocation");
    float* d_sc = (float*)((char*)d + bx);
    cudaError_t e = cudaMemcpy(d, x, (size_t)n * sizeof(float), cudaMemcpyHostToDevice);
    if (e == cudaSuccess) e = launch_trig_eval(d, d_sc, (long long)n, 0);
    if (e == cudaSuccess) e = cudaMemcpy(sincos, d_sc, (size_t)n * 2 * sizeof(float), cudaMemcpyDeviceToHost);
    cudaFree(d);
    CUDA_OR_FAIL(e, "trig eval");
    return RLC_OK;
}

int rlc_count_steps(rlc_method* m, const float* ins, const float* angles, int n, int na, unsigned flags,
                    int64_t* total_steps) {
    if (int rc = check_method(m)) return rc;
    if (!total_steps) return fail(RLC_ERR_ARG, "null output");
    if (m->dkind == K_CDDT || m->dkind == K_GLT) return fail(RLC_ERR_STATE, "step counts apply to RM and BL");
    if (n < 0 || na < 0) return fail(RLC_ERR_ARG, "negative size");
    *total_steps = 0;
    if ((long long)n * na == 0) return RLC_OK;
    if (!ins || !angles) return fail(RLC_ERR_ARG, "null array");
    if (int rc = check_trig(m, (long long)n * na)) return rc;
    CastParams p = m->params();
    p.map.dt = m->map->d_dt;   // the counting kernel marches the linear distance transform whatever the schedule
    const float* d_in = ins;
    const float* d_ang = angles;
    void* st = nullptr;
    size_t b0 = align256((size_t)n * 3 * sizeof(float)), b1 = align256((size_t)na * sizeof(float));
    if (int rc = m->stage(b0 + b1 + sizeof(unsigned long long), &st)) return rc;
    unsigned long long* d_total = (unsigned long long*)((char*)st + b0 + b1);
    if (!(flags & RLC_DEVICE_PTRS)) {
        CUDA_OR_FAIL(cudaMemcpy(st, ins, (size_t)n * 3 * sizeof(float), cudaMemcpyHostToDevice), "H2D");
        CUDA_OR_FAIL(cudaMemcpy((char*)st + b0, angles, (size_t)na * sizeof(float), cudaMemcpyHostToDevice), "H2D");
        d_in = (const float*)st;
        d_ang = (const float*)((char*)st + b0);
    }
    CUDA_OR_FAIL(cudaMemset(d_total, 0, sizeof(unsigned long long)), "count steps");
    CUDA_OR_FAIL(launch_count_steps(p, d_in, d_ang, n, na, d_total, 0), "count steps");
    unsigned long long tot = 0;
    CUDA_OR_FAIL(cudaMemcpy(&tot, d_total, sizeof(tot), cudaMemcpyDeviceToHost), "count steps");
    *total_steps = (int64_t)tot;
    return RLC_OK;
}

int rlc_method_set_schedule(rlc_method* m, int dt_layout, int fused_block, int prefetch, int tile) {
    if (int rc = check_method(m)) return rc;
    if (dt_layout < -1 || dt_layout > 5) return fail(RLC_ERR_ARG, "dt_layout must be -1, 0, 1, 2, 3, 4 or 5");
    if (fused_block != 0 && (fused_block < 32 || fused_block > 512 || fused_block % 32))
        return fail(RLC_ERR_ARG, "fused_block must be a multiple of 32 in [32, 512]");
    if (prefetch < 0 || prefetch > (m->dkind == K_CDDT ? 2 : 1))
        return fail(RLC_ERR_ARG, m->dkind == K_CDDT ? "prefetch must be 0, 1 or 2" : "prefetch must be 0 or 1");
    if (tile < 0 || tile > 512) return fail(RLC_ERR_ARG, "tile must be in [0, 512]");
    if (dt_layout == -1) {
        m->autotune_pending = true;
    } else {
        m->layout = dt_layout;
        m->prefetch = prefetch;
        m->tile = tile;
        m->pick = m->pick_fused = false;
    }
    if (fused_block) m->fused_block = fused_block;
    return RLC_OK;
}

int rlc_method_get_schedule(const rlc_method* m, int* dt_layout, int* fused_block, int* prefetch, int* tile) {
    if (int rc = check_method(m)) return rc;
    if (dt_layout) *dt_layout = m->layout;
    if (fused_block) *fused_block = m->fused_block;
    if (prefetch) *prefetch = m->prefetch;
    if (tile) *tile = m->tile;
    return RLC_OK;
}

constexpr int kTuneFirst = 5;       // stage 1: timed launches per candidate (median)
constexpr int kTuneFinal = 31;      // stage 2: timed launches per finalist, round-robin (median)
constexpr int kTuneFinalists = 3;

static float median_of(std::vector<float> v) {
    if (v.empty()) return 1e30f;
    std::sort(v.begin(), v.end());
    return v[v.size() / 2];
}

// Times every schedule candidate (distance-transform layout x RM march variant or CDDT bin search
// x block size x particles per tile, the staged update, and what the call picks without a schedule) on the caller's workload with CUDA
// events around single launches: the median of kTuneFirst launches for every candidate, then the
// median of kTuneFinal launches for the kTuneFinalists fastest, taken round-robin so that clock
// and neighbour drift falls on all of them alike.  With RLC_TUNE_FLUSH_L2 a write of twice the
// L2 size precedes every timed launch (a device buffer held for the duration of the call).
int rlc_method_autotune_ex(rlc_method* m, const float* ins, const float* angles, const float* obs, double* w, int n,
                           int na, unsigned flags, void* stream) {
    if (int rc = check_method(m)) return rc;
    if (!m->d_table) return fail(RLC_ERR_STATE, "set_sensor_model has not been called");
    if (n <= 0) return RLC_OK;
    cudaStream_t s = (cudaStream_t)stream;
    using Cand = rlc_method::TuneResult;
    std::vector<Cand> cands;
    const int blocks[3] = {128, 256, 512};
    const int tiles[3] = {0, 16, 32};
    const bool rm = m->dkind == K_RM;
    static const int kLayouts[5] = {DT_LINEAR, DT_TILED, DT_U16, DT_STEP, DT_RUNS};
    for (int lk = 0; lk < (rm ? 5 : 1); ++lk)
        // march variants: RM plain / prefetching; CDDT binary / sector search
        for (int pk = 0; pk < (rm || m->dkind == K_CDDT ? 2 : 1); ++pk)
            for (int bi = 0; bi < 3; ++bi)
                for (int ti = 0; ti < 3; ++ti) {
                    if (ti > 0 && tile_particles(na, blocks[bi], tiles[ti]) == tile_particles(na, blocks[bi], 0))
                        continue;   // same tile as the automatic choice
                    const int pf = (m->dkind == K_CDDT && pk) ? 2 : pk;
                    cands.push_back(Cand{{kLayouts[lk], blocks[bi], pf, tiles[ti], false}, 0.0f, 0.0f});
                }
    if (rm) {   // beam-major update with staged windows
        if (int rc = ensure_bins(m, (size_t)n * na)) return rc;
        cands.push_back(Cand{{DT_STAGED, 0, 0, 0, false}, 0.0f, 0.0f});
    }
    cands.push_back(Cand{{picked_fused_layout(m, n, na), 0, 0, 0, true}, 0.0f, 0.0f});   // the call's own choice
    void* flush = nullptr;
    size_t flush_bytes = 0;
    if (flags & RLC_TUNE_FLUSH_L2) {
        int dev = 0, l2 = 0;
        CUDA_OR_FAIL(cudaGetDevice(&dev), "autotune");
        CUDA_OR_FAIL(cudaDeviceGetAttribute(&l2, cudaDevAttrL2CacheSize, dev), "autotune");
        flush_bytes = 2 * (size_t)(l2 > 0 ? l2 : (64 << 20));
        if (cudaMalloc(&flush, flush_bytes) != cudaSuccess) {
            cudaGetLastError();
            return fail(RLC_ERR_NOMEM, "autotune: no room for the %zu-byte L2 flush buffer", flush_bytes);
        }
    }
    cudaEvent_t e0 = nullptr, e1 = nullptr;
    cudaError_t err = cudaEventCreate(&e0);
    if (err == cudaSuccess) err = cudaEventCreate(&e1);
    auto launch = [&](const Cand& c) { return launch_fused_as(m, c.f, ins, angles, obs, w, n, na, s); };
    unsigned flush_round = 0;
    auto time_once = [&](const Cand& c, float* ms) -> cudaError_t {
        cudaError_t e = cudaSuccess;
        if (flush) e = cudaMemsetAsync(flush, (int)(++flush_round & 0xFF), flush_bytes, s);
        if (e == cudaSuccess) e = cudaEventRecord(e0, s);
        if (e == cudaSuccess) e = launch(c);
        if (e == cudaSuccess) e = cudaEventRecord(e1, s);
        if (e == cudaSuccess) e = cudaEventSynchronize(e1);
        if (e == cudaSuccess) e = cudaEventElapsedTime(ms, e0, e1);
        return e;
    };
    for (size_t i = 0; i < cands.size() && err == cudaSuccess; ++i) {
        err = launch(cands[i]);   // warm-up (first use of the variant)
        std::vector<float> t;
        for (int r = 0; r < kTuneFirst && err == cudaSuccess; ++r) {
            float ms = 0.0f;
            err = time_once(cands[i], &ms);
            t.push_back(ms);
        }
        cands[i].first_ms = median_of(t);
    }
    std::vector<int> order(cands.size());
    for (size_t i = 0; i < order.size(); ++i) order[i] = (int)i;
    std::sort(order.begin(), order.end(), [&](int a, int b) { return cands[a].first_ms < cands[b].first_ms; });
    const int nf = (int)std::min<size_t>(kTuneFinalists, order.size());
    std::vector<std::vector<float>> fin(nf);
    for (int r = 0; r < kTuneFinal && err == cudaSuccess; ++r)
        for (int k = 0; k < nf && err == cudaSuccess; ++k) {
            float ms = 0.0f;
            err = time_once(cands[order[k]], &ms);
            fin[k].push_back(ms);
        }
    int best = order.empty() ? -1 : order[0];
    float best_ms = 1e30f;
    for (int k = 0; k < nf; ++k) {
        cands[order[k]].final_ms = median_of(fin[k]);
        if (cands[order[k]].final_ms < best_ms) {
            best_ms = cands[order[k]].final_ms;
            best = order[k];
        }
    }
    if (e0) cudaEventDestroy(e0);
    if (e1) cudaEventDestroy(e1);
    if (flush) cudaFree(flush);
    if (err != cudaSuccess) return cuda_fail(err, "autotune");
    if (best >= 0) {
        const rlc_method::Fused& b = cands[best].f;
        m->pick_fused = b.pick;
        m->layout = b.layout;
        if (b.block) m->fused_block = b.block;
        m->prefetch = b.prefetch;
        m->tile = b.tile;
    }
    m->tune_results = cands;
    return RLC_OK;
}

int rlc_method_autotune(rlc_method* m, const float* ins, const float* angles, const float* obs, double* w, int n,
                        int na, void* stream) {
    return rlc_method_autotune_ex(m, ins, angles, obs, w, n, na, 0, stream);
}

int rlc_method_autotune_results(const rlc_method* m, int max, int* count, int* schedules, float* times_ms) {
    if (int rc = check_method(m)) return rc;
    if (!count) return fail(RLC_ERR_ARG, "null output");
    *count = (int)m->tune_results.size();
    for (int i = 0; i < max && i < *count; ++i) {
        const auto& r = m->tune_results[i];
        if (schedules) {
            schedules[4 * i] = r.f.layout;
            schedules[4 * i + 1] = r.f.block;
            schedules[4 * i + 2] = r.f.prefetch;
            schedules[4 * i + 3] = r.f.tile;
        }
        if (times_ms) {
            times_ms[2 * i] = r.first_ms;
            times_ms[2 * i + 1] = r.final_ms;
        }
    }
    return RLC_OK;
}

}  // extern "C"

// ============================================================ batched filters
struct rlc_batch {
    std::vector<rlc_filter_desc> descs;
    bool rm_only = true;
    // schedule
    int layout = DT_LINEAR, prefetch = 0, block = 256, tile = 0;
    bool separate = false;    // products in a second launch instead of inside the persistent kernel
    // nothing asked for or autotuned yet: a batch of ray-marching filters runs with the products
    // inside the launch (k_batch_wide), on the step map with its equal-step runs while the run waits
    // for its longest rays (below 2 M rays: one filter of 1,198 x 120 36 against 51 us without), and
    // the getters report the values above meanwhile.  8 filters of 512^2 - 4096^2, 23 M rays: those
    // values 987 us, the best schedule of k_batch 649, this 575.  From 48 M rays on, that schedule of
    // k_batch, whose march budget gains what its second launch costs: 45 M rays 1003 against 1012 us,
    // 73 M 1504 / 1577, 122 M 2529 / 2772.
    bool pick = true;
    struct Schedule { int layout, prefetch, block, tile; bool separate, wide; } run{};   // what is run
    // built state
    int nf = 0;
    FilterDev* d_filters = nullptr;
    unsigned* d_queue = nullptr;
    uint16_t* d_bins = nullptr;   // every filter's range bins, tile by tile (batch_tile_bins)
    size_t bins_cap = 0;          // entries of d_bins
    uint16_t* d_obs_bins = nullptr;   // every filter's observation bins
    float4* d_rec = nullptr;          // every filter's particle and beam records (FilterDev::part_rec, beam_rec)
    unsigned total_tiles = 0;
    unsigned total_particles = 0;
    long long rays = 0;
    int grid = 0;
    size_t smem = 0;
    cudaStream_t cap = nullptr;
    cudaGraph_t graph = nullptr;
    cudaGraphExec_t exec = nullptr;
    std::vector<unsigned> seen;   // each method's generation in the device table; empty: no table

    void drop_graph() {
        if (exec) cudaGraphExecDestroy(exec);
        if (graph) cudaGraphDestroy(graph);
        exec = nullptr;
        graph = nullptr;
    }
    ~rlc_batch() {
        drop_graph();
        if (cap) cudaStreamDestroy(cap);
        cudaFree(d_filters);
        cudaFree(d_queue);
        cudaFree(d_bins);
        cudaFree(d_obs_bins);
        cudaFree(d_rec);
    }

    // (re)build the device filter table for the current schedule
    int build() {
        drop_graph();
        seen.clear();
        for (size_t i = 0; i < descs.size(); ++i) {
            const rlc_method* m = descs[i].method;
            if (!m->d_table) return fail(RLC_ERR_STATE, "filter %d: sensor model not set", (int)i);
            if (m->d_trig && m->trig_count < (long long)descs[i].n_particles * descs[i].n_angles)
                return fail(RLC_ERR_ARG, "filter %d: trig override too short", (int)i);
        }
        if (d_filters) CUDA_OR_FAIL(cudaDeviceSynchronize(), "batch setup");   // a run may still be reading the table
        int dev = 0, sms = 0;
        CUDA_OR_FAIL(cudaGetDevice(&dev), "batch setup");
        CUDA_OR_FAIL(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev), "batch setup");
        run = Schedule{layout, prefetch, block, tile, separate, false};
        bool steps = true;   // every ray-marching filter's map has a step map
        long long particles = 0, run_rays = 0;   // rays on maps with long equal-step runs
        for (const rlc_filter_desc& d : descs) {
            if (d.method->dkind == K_RM && map_layout(d.method->map, DT_STEP) != DT_STEP) steps = false;
            particles += d.n_particles;
            if (d.method->map->long_runs) run_rays += (long long)d.n_particles * d.n_angles;
        }
        if (!steps && (layout == DT_STEP || layout == DT_RUNS)) run.layout = DT_LINEAR;
        if (pick && rm_only && steps) {
            if (rays < (48ll << 20))
                run = Schedule{rays < (2ll << 20) && 2 * run_rays >= rays ? DT_RUNS : DT_STEP, 0, 256, batch_wide_tile(particles, sms), false, true};
            else
                run = Schedule{DT_STEP, 0, 256, 8, true, false};
        }
        struct Item { FilterDev f; double cost; };
        std::vector<Item> items;
        const int ppb = run.tile > 0 ? run.tile : 32;   // 32 particles: one full lane set of the product warp
        size_t need = 0, nobs = 0, nrec = 0;
        for (const rlc_filter_desc& d : descs) {
            if (run.wide) break;   // no bins, no records
            need += (size_t)((d.n_particles + ppb - 1) / ppb) * batch_tile_bins(d.n_angles, ppb);
            nobs += (size_t)d.n_angles;
            nrec += 2 * (size_t)d.n_particles + (size_t)d.n_angles;
        }
        if (need > bins_cap) {
            cudaFree(d_bins);
            d_bins = nullptr;
            bins_cap = 0;
            CUDA_OR_FAIL(cudaMalloc(&d_bins, (need ? need : 1) * sizeof(uint16_t)), "batch range bins");
            bins_cap = need;
        }
        if (!run.wide && !d_obs_bins) CUDA_OR_FAIL(cudaMalloc(&d_obs_bins, (nobs ? nobs : 1) * sizeof(uint16_t)), "batch observation bins");
        if (!run.wide && !d_rec) CUDA_OR_FAIL(cudaMalloc(&d_rec, (nrec ? nrec : 1) * sizeof(float4)), "batch particle and beam records");
        size_t bin_ofs = 0, obs_ofs = 0, rec_ofs = 0;
        for (const rlc_filter_desc& d : descs) {
            rlc_method* m = d.method;
            Item it{};
            CastParams p = m->params();
            if (m->dkind == K_RM) {   // the batch schedule's layout for every ray-marching filter
                p.map.dt = run.layout == DT_TILED ? m->map->d_dt_tiled : m->map->d_dt;
            }
            it.f.p = p;
            it.f.layout = run.layout;
            it.f.prefetch = run.prefetch;
            it.f.sm = SensorDev{m->d_table, m->K};
            it.f.ins = d.ins;
            it.f.angles = d.angles;
            it.f.obs = d.obs;
            it.f.ranges = d.ranges;
            it.f.weights = d.weights;
            it.f.n = d.n_particles;
            it.f.na = d.n_angles;
            it.f.inv_na = d.n_angles > 0 ? 1.0f / (float)d.n_angles : 0.0f;
            it.f.ppb = ppb;
            if (!run.wide) {
                it.f.bins = d_bins + bin_ofs;
                bin_ofs += (size_t)((d.n_particles + ppb - 1) / ppb) * batch_tile_bins(d.n_angles, ppb);
                it.f.obs_bins = d_obs_bins + obs_ofs;
                obs_ofs += (size_t)d.n_angles;
                it.f.part_rec = d_rec + rec_ofs;
                rec_ofs += 2 * (size_t)d.n_particles;
                it.f.beam_rec = d_rec + rec_ofs;
                rec_ofs += (size_t)d.n_angles;
            }
            // heavier tiles first: rays per tile x march length
            it.cost = (double)it.f.ppb * (d.n_angles > 0 ? d.n_angles : 1) * (double)(m->mr > 1.0f ? m->mr : 1.0f);
            items.push_back(it);
        }
        std::stable_sort(items.begin(), items.end(), [](const Item& a, const Item& b) { return a.cost > b.cost; });
        unsigned long long tiles = 0, parts = 0;
        std::vector<FilterDev> hf;
        for (auto& it : items) {
            it.f.part_begin = (unsigned)parts;
            parts += (unsigned long long)it.f.n;
            if (parts >= 0xffffffffull) return fail(RLC_ERR_ARG, "too many particles in one batch");
            it.f.tile_begin = (unsigned)tiles;
            tiles += (unsigned long long)((it.f.n + it.f.ppb - 1) / it.f.ppb);
            if (tiles >= 0xffffffffull) return fail(RLC_ERR_ARG, "too many tiles in one batch");
            hf.push_back(it.f);
        }
        int per_sm = 0;
        cudaError_t e = cudaSuccess;
        smem = batch_smem(run.block, rm_only);
        if (run.wide) e = batch_wide_occupancy(run.layout, run.tile, &per_sm);
        else
            e = batch_occupancy(run.block, smem, rm_only, run.layout, run.prefetch, run.separate, &per_sm);
        if (e == cudaSuccess && per_sm <= 0) e = cudaErrorInvalidConfiguration;
        if (e == cudaSuccess && !d_filters) e = cudaMalloc(&d_filters, descs.size() * sizeof(FilterDev));
        if (e == cudaSuccess)
            e = cudaMemcpy(d_filters, hf.data(), hf.size() * sizeof(FilterDev), cudaMemcpyHostToDevice);
        if (e == cudaSuccess && !d_queue) e = cudaMalloc(&d_queue, sizeof(unsigned));
        if (e == cudaSuccess && !cap) e = cudaStreamCreateWithFlags(&cap, cudaStreamNonBlocking);
        if (e != cudaSuccess) return cuda_fail(e, "batch setup");
        nf = (int)hf.size();
        total_tiles = (unsigned)tiles;
        total_particles = (unsigned)parts;
        long long g = (long long)sms * per_sm;
        if (g > (long long)tiles) g = (long long)tiles;
        grid = (int)(g > 0 ? g : 1);
        for (const rlc_filter_desc& d : descs) seen.push_back(d.method->generation);
        return RLC_OK;
    }

    // queue reset + persistent kernel, captured once as a CUDA graph
    int launch(cudaStream_t stream) {
        if (total_tiles == 0) return RLC_OK;
        // a method whose trig override, sensor model or CDDT table was replaced since the build: the device
        // table holds the old (freed) one, so rebuild it (and the graph) first
        bool current = !seen.empty();
        for (size_t i = 0; i < seen.size(); ++i) current = current && descs[i].method->generation == seen[i];
        if (!current)
            if (int rc = build()) return rc;
        if (!exec) {
            CUDA_OR_FAIL(cudaStreamBeginCapture(cap, cudaStreamCaptureModeThreadLocal), "batch capture");
            cudaError_t e = cudaMemsetAsync(d_queue, 0, sizeof(unsigned), cap);
            if (e == cudaSuccess && run.wide)
                e = launch_batch_wide(d_filters, nf, total_tiles, d_queue, grid, run.layout, run.tile, cap);
            else if (e == cudaSuccess)
                e = launch_batch(d_filters, nf, total_tiles, d_queue, grid, run.block, smem, rm_only, run.layout,
                                 run.prefetch, run.separate, total_particles, cap);
            cudaGraph_t g = nullptr;
            cudaError_t e2 = cudaStreamEndCapture(cap, &g);
            if (e == cudaSuccess) e = e2;
            if (e == cudaSuccess) e = cudaGraphInstantiate(&exec, g, 0);
            if (e != cudaSuccess) {
                if (g) cudaGraphDestroy(g);
                exec = nullptr;
                return cuda_fail(e, "batch graph");
            }
            graph = g;
        }
        CUDA_OR_FAIL(cudaGraphLaunch(exec, stream), "batch launch");
        return RLC_OK;
    }
};

extern "C" {

int rlc_batch_create(const rlc_filter_desc* fd, int nf, int block, rlc_batch** out) {
    if (!out) return fail(RLC_ERR_ARG, "null output handle");
    *out = nullptr;
    if (nf <= 0 || !fd) return fail(RLC_ERR_ARG, "a batch needs at least one filter");
    const bool asked = block != 0;
    if (!asked) block = 256;
    if (block < 32 || block > 512 || block % 32) return fail(RLC_ERR_ARG, "block must be a multiple of 32 in [32, 512]");
    long long rays = 0;
    bool rm_only = true;
    for (int i = 0; i < nf; ++i) {
        const rlc_filter_desc& d = fd[i];
        rlc_method* m = d.method;
        if (!m) return fail(RLC_ERR_ARG, "filter %d: null method", i);
        if (d.n_particles < 0 || d.n_angles < 0) return fail(RLC_ERR_ARG, "filter %d: negative size", i);
        if (d.n_angles > 16384) return fail(RLC_ERR_ARG, "filter %d: at most 16384 beams", i);
        if (d.n_particles > 0 && (!d.ins || !d.weights || (d.n_angles > 0 && (!d.angles || !d.obs))))
            return fail(RLC_ERR_ARG, "filter %d: null array", i);
        if ((long long)d.n_particles * d.n_angles > (1ll << 31) - 1) return fail(RLC_ERR_ARG, "filter %d: too many rays", i);
        rays += (long long)d.n_particles * d.n_angles;
        if (m->dkind != K_RM) rm_only = false;
    }
    rlc_batch* b = new rlc_batch();
    b->descs.assign(fd, fd + nf);
    b->rm_only = rm_only;
    b->block = block;
    b->pick = !asked;
    b->rays = rays;
    if (int rc = b->build()) {
        delete b;
        return rc;
    }
    *out = b;
    return RLC_OK;
}

int rlc_batch_set_schedule(rlc_batch* b, int dt_layout, int prefetch, int block, int tile) {
    if (!b) return fail(RLC_ERR_ARG, "null batch handle");
    if (dt_layout < 0 || dt_layout > 5 || dt_layout == DT_STAGED)
        return fail(RLC_ERR_ARG, "dt_layout must be 0, 1, 2, 4 or 5");
    if (prefetch < 0 || prefetch > 1) return fail(RLC_ERR_ARG, "prefetch must be 0 or 1");
    if (block != 0 && (block < 32 || block > 512 || block % 32)) return fail(RLC_ERR_ARG, "block must be a multiple of 32 in [32, 512]");
    if (tile < 0 || tile > 512) return fail(RLC_ERR_ARG, "tile must be in [0, 512]");
    b->pick = false;
    b->layout = dt_layout;
    b->prefetch = prefetch;
    if (block) b->block = block;
    b->tile = tile;
    return b->build();
}

int rlc_batch_set_product_mode(rlc_batch* b, int mode) {
    if (!b) return fail(RLC_ERR_ARG, "null batch handle");
    if (mode != RLC_PRODUCTS_OVERLAPPED && mode != RLC_PRODUCTS_SEPARATE) return fail(RLC_ERR_ARG, "product mode %d", mode);
    b->pick = false;
    b->separate = mode == RLC_PRODUCTS_SEPARATE;
    return b->build();
}

int rlc_batch_get_product_mode(const rlc_batch* b, int* mode) {
    if (!b || !mode) return fail(RLC_ERR_ARG, "null argument");
    *mode = b->separate ? RLC_PRODUCTS_SEPARATE : RLC_PRODUCTS_OVERLAPPED;
    return RLC_OK;
}

int rlc_batch_get_schedule(const rlc_batch* b, int* dt_layout, int* prefetch, int* block, int* tile) {
    if (!b) return fail(RLC_ERR_ARG, "null batch handle");
    if (dt_layout) *dt_layout = b->layout;
    if (prefetch) *prefetch = b->prefetch;
    if (block) *block = b->block;
    if (tile) *tile = b->tile;
    return RLC_OK;
}

// Runs the batch under each schedule candidate (outputs are overwritten with
// identical values), keeps the fastest.
// Runs the batch under each schedule candidate (outputs are overwritten with identical values):
// every candidate timed over two launches after a warm-up, then the three fastest re-timed
// round-robin over 9 launches each (median); keeps the fastest.
int rlc_batch_autotune(rlc_batch* b, void* stream) {
    if (!b) return fail(RLC_ERR_ARG, "null batch handle");
    cudaStream_t s = (cudaStream_t)stream;
    struct Cand { bool sep; int layout, pf, block, tile; float ms; bool pick; };
    std::vector<Cand> cands;
    const int blocks[2] = {256, 512};
    const int tiles[3] = {8, 16, 32};
    static const int kLayouts[5] = {DT_LINEAR, DT_TILED, DT_U16, DT_STEP, DT_RUNS};
    for (int sp = 0; sp < 2; ++sp)
        for (int lk = 0; lk < 5; ++lk)
            for (int pf = 0; pf < 2; ++pf)
                for (int bi = 0; bi < 2; ++bi)
                    for (int ti = 0; ti < 3; ++ti) {
                        if (!b->rm_only && (kLayouts[lk] != 0 || pf != 0)) continue;
                        cands.push_back(Cand{sp != 0, kLayouts[lk], pf, blocks[bi], tiles[ti], 0.0f, false});
                    }
    if (b->rm_only) {   // the batch's own choice: the wide launch, where it comes to that
        const bool pick = b->pick;
        b->pick = true;
        const int rc = b->build();
        b->pick = pick;
        if (rc) return rc;
        const rlc_batch::Schedule& r = b->run;
        if (r.wide) cands.push_back(Cand{r.separate, r.layout, r.prefetch, r.block, r.tile, 0.0f, true});
    }
    const bool s0 = b->separate, pick0 = b->pick;
    const int l0 = b->layout, p0 = b->prefetch, b0 = b->block, t0 = b->tile;
    auto apply = [&](const Cand& c) {
        b->pick = c.pick;
        b->separate = c.sep;
        b->layout = c.layout;
        b->prefetch = c.pf;
        b->block = c.block;
        b->tile = c.tile;
        return b->build();
    };
    cudaEvent_t e0 = nullptr, e1 = nullptr;
    int rc = RLC_OK;
    if (cudaEventCreate(&e0) != cudaSuccess || cudaEventCreate(&e1) != cudaSuccess) rc = cuda_fail(cudaGetLastError(), "batch autotune");
    auto time_launches = [&](int reps, float* ms) -> int {
        if (int r = b->launch(s)) return r;   // warm (and graph capture)
        cudaEventRecord(e0, s);
        for (int rep = 0; rep < reps; ++rep)
            if (int r = b->launch(s)) return r;
        cudaEventRecord(e1, s);
        cudaError_t e = cudaEventSynchronize(e1);
        if (e == cudaSuccess) e = cudaEventElapsedTime(ms, e0, e1);
        if (e != cudaSuccess) return cuda_fail(e, "batch autotune");
        *ms /= (float)reps;
        return RLC_OK;
    };
    for (size_t i = 0; i < cands.size() && !rc; ++i) {
        if ((rc = apply(cands[i]))) break;
        rc = time_launches(2, &cands[i].ms);
    }
    std::vector<int> order(cands.size());
    for (size_t i = 0; i < order.size(); ++i) order[i] = (int)i;
    std::sort(order.begin(), order.end(), [&](int a, int c) { return cands[a].ms < cands[c].ms; });
    const int nf = (int)std::min<size_t>(3, order.size());
    std::vector<std::vector<float>> fin(nf);
    for (int r = 0; r < 9 && !rc; ++r)
        for (int k = 0; k < nf && !rc; ++k) {
            float ms = 0.0f;
            if ((rc = apply(cands[order[k]]))) break;
            rc = time_launches(1, &ms);
            fin[k].push_back(ms);
        }
    int best = -1;
    float best_ms = 1e30f;
    for (int k = 0; k < nf && !rc; ++k) {
        const float med = median_of(fin[k]);
        if (med < best_ms) {
            best_ms = med;
            best = order[k];
        }
    }
    if (e0) cudaEventDestroy(e0);
    if (e1) cudaEventDestroy(e1);
    if (best >= 0) {
        int rc2 = apply(cands[best]);
        return rc ? rc : rc2;
    }
    b->pick = pick0;
    b->separate = s0;
    b->layout = l0;
    b->prefetch = p0;
    b->block = b0;
    b->tile = t0;
    int rc2 = b->build();
    return rc ? rc : rc2;
}

int rlc_batch_run(rlc_batch* b, void* stream) {
    if (!b) return fail(RLC_ERR_ARG, "null batch handle");
    return b->launch((cudaStream_t)stream);
}

int rlc_batch_destroy(rlc_batch* b) {
    delete b;
    return RLC_OK;
}

int rlc_batch_info(const rlc_batch* b, int64_t* rays, int64_t* tiles) {
    if (!b) return fail(RLC_ERR_ARG, "null batch handle");
    if (rays) *rays = b->rays;
    if (tiles) *tiles = b->total_tiles;
    return RLC_OK;
}

}  // extern "C"
