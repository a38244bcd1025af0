// The library's host code on a stand-in for the CUDA runtime: every runtime function that
// librangelibc_gb300.so imports is defined here, so that no GPU is needed and none is touched.
// "Device" memory is host memory that is filled with ones and never given back (a pointer into a freed
// block stays recognisable), kernels do not run but are recorded, allocations can be made to fail, and
// a kernel's time is what the scenario says.
//
//   host_calls <scenario>     prints "ok", or what was wrong, and exits non-zero then
#include "rangelibc.h"

#include <cuda_runtime_api.h>
#include <cxxabi.h>

#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <functional>
#include <map>
#include <string>
#include <vector>

namespace {

struct Block { size_t bytes; bool live; };
std::map<char*, Block> blocks;                    // by address, freed ones too
std::map<const void*, std::string>& kernels() {   // host function -> demangled name; filled before this file's own globals are made
    static std::map<const void*, std::string> m;
    return m;
}
size_t refuse_from = ~(size_t)0;                  // allocations of this many bytes or more fail
long long calls = 0;                              // runtime calls of any kind
std::function<void(const std::string&, void**)> on_launch = [](const std::string&, void**) {};
std::function<float(const std::string&)> kernel_ms = [](const std::string&) { return 1.0f; };
float clock_ms = 0.0f;
std::map<cudaEvent_t, float> events;
std::map<const void*, int> smem_limit;
int lowered = 0;                                  // times a kernel's shared-memory limit went down

std::map<void*, bool> in_flight;                  // blocks that a launched graph may still be reading
int torn = 0;                                     // copies into one of them

struct Launch { std::string name; std::vector<void*> words; };   // the first parameter, where it is a pointer
bool capturing = false;
std::vector<Launch> recorded;

std::string last_kernel;

void launched(const void* f, void** args) {
    const std::string& name = last_kernel = kernels()[f];
    clock_ms += kernel_ms(name);
    on_launch(name, args);
    if (capturing) recorded.push_back(Launch{name, {args ? *(void**)args[0] : nullptr}});
}

// the words of the block at p that point into freed memory
int stale_words(void* p) {
    auto it = blocks.find((char*)p);
    if (it == blocks.end()) return 0;
    int n = 0;
    for (size_t i = 0; i + sizeof(char*) <= it->second.bytes; i += sizeof(char*)) {
        char* w;
        memcpy(&w, it->first + i, sizeof(w));
        auto at = blocks.upper_bound(w);
        if (at == blocks.begin()) continue;
        --at;
        if (!at->second.live && w < at->first + at->second.bytes) ++n;
    }
    return n;
}

}  // namespace

extern "C" {
cudaError_t cudaMalloc(void** p, size_t n) {
    ++calls;
    *p = nullptr;
    if (n >= refuse_from) return cudaErrorMemoryAllocation;
    char* b = (char*)aligned_alloc(256, (n + 255) / 256 * 256);
    memset(b, 1, n);
    blocks[b] = Block{n, true};
    *p = b;
    return cudaSuccess;
}
cudaError_t cudaFree(void* p) {
    ++calls;
    if (p) {
        blocks[(char*)p].live = false;
        in_flight.clear();   // waits for the device
    }
    return cudaSuccess;
}
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind) {
    ++calls;
    torn += (int)in_flight.count(d);   // (not ordered with streams that do not wait for the legacy one)
    memcpy(d, s, n);
    return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t) { ++calls; memcpy(d, s, n); return cudaSuccess; }
cudaError_t cudaMemset(void* d, int v, size_t n) { ++calls; memset(d, v, n); return cudaSuccess; }
cudaError_t cudaMemsetAsync(void* d, int v, size_t n, cudaStream_t) { ++calls; memset(d, v, n); return cudaSuccess; }
cudaError_t cudaGetLastError(void) { return cudaSuccess; }
const char* cudaGetErrorString(cudaError_t) { return "stand-in error"; }
cudaError_t cudaGetDevice(int* d) { ++calls; *d = 0; return cudaSuccess; }
cudaError_t cudaSetDevice(int) { ++calls; return cudaSuccess; }
cudaError_t cudaGetDeviceCount(int* n) { *n = 1; return cudaSuccess; }
cudaError_t cudaDeviceSynchronize(void) { ++calls; in_flight.clear(); return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr a, int) {
    *v = a == cudaDevAttrMultiProcessorCount ? 152 : a == cudaDevAttrL2CacheSize ? 1 << 20 : a == cudaDevAttrPageableMemoryAccess;
    return cudaSuccess;
}
cudaError_t cudaEventCreate(cudaEvent_t* e) { *e = (cudaEvent_t)malloc(1); return cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t) { events[e] = clock_ms; return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t a, cudaEvent_t b) { *ms = events[b] - events[a]; return cudaSuccess; }
cudaError_t cudaFuncSetAttribute(const void* f, cudaFuncAttribute a, int v) {
    ++calls;
    if (a == cudaFuncAttributeMaxDynamicSharedMemorySize) {
        if (smem_limit.count(f) && v < smem_limit[f]) ++lowered;
        smem_limit[f] = v;
    }
    return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int* n, const void*, int, size_t, unsigned) { *n = 4; return cudaSuccess; }
// cuTensorMapEncodeTiled
static int encode(void*, int, unsigned, void*, const void*, const void*, const unsigned*, const unsigned*, int, int, int, int) {
    return 0;
}
cudaError_t cudaGetDriverEntryPointByVersion(const char*, void** p, unsigned, unsigned long long, cudaDriverEntryPointQueryResult* q) {
    *p = (void*)encode;
    *q = cudaDriverEntryPointSuccess;
    return cudaSuccess;
}
cudaError_t cudaGetSymbolAddress(void** p, const void*) { return cudaMalloc(p, 1024); }
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes* a, const void*) { memset(a, 0, sizeof(*a)); return cudaSuccess; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) { *s = (cudaStream_t)malloc(1); return cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { ++calls; return cudaSuccess; }
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) { capturing = true; recorded.clear(); return cudaSuccess; }
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t* g) {
    capturing = false;
    *g = (cudaGraph_t) new std::vector<Launch>(recorded);
    return cudaSuccess;
}
cudaError_t cudaGraphInstantiate(cudaGraphExec_t* e, cudaGraph_t g, unsigned long long) {
    *e = (cudaGraphExec_t) new std::vector<Launch>(*(std::vector<Launch>*)g);
    return cudaSuccess;
}
cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }
static std::vector<Launch> last_graph;
cudaError_t cudaGraphLaunch(cudaGraphExec_t e, cudaStream_t) {
    last_graph = *(std::vector<Launch>*)e;
    for (const Launch& l : last_graph) {
        clock_ms += kernel_ms(l.name);
        in_flight[l.words[0]] = true;
    }
    return cudaSuccess;
}
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t*, const void* f, void** args) { ++calls; launched(f, args); return cudaSuccess; }
// what nvcc's host code calls to register and launch kernels
cudaError_t __cudaGetKernel(void** k, const void* f) { *k = (void*)f; return cudaSuccess; }
cudaError_t __cudaLaunchKernel(void* k, dim3, dim3, void** args, size_t, cudaStream_t) { ++calls; launched(k, args); return cudaSuccess; }
unsigned __cudaPushCallConfiguration(dim3, dim3, size_t, cudaStream_t) { return 0; }
cudaError_t __cudaPopCallConfiguration(dim3*, dim3*, size_t*, void*) { return cudaSuccess; }
void** __cudaRegisterFatBinary(void*) { static void* h; return &h; }
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterVar(void**, char*, char*, const char*, int, size_t, int, int) {}
void __cudaRegisterFunction(void**, const char* f, char*, const char* name, int, void*, void*, void*, void*, int*) {
    int st = 0;
    char* d = abi::__cxa_demangle(name, nullptr, nullptr, &st);
    kernels()[f] = d ? d : name;
    free(d);
}
}

namespace {

int wrong(const char* what) {
    printf("%s (%s)\n", what, rlc_last_error());
    return 1;
}
#define CHECK(c) do { if (!(c)) return wrong(#c); } while (0)

rlc_method* method(int kind, int W = 64, int H = 48, unsigned td = 0) {
    std::vector<uint8_t> occ((size_t)W * H, 0);
    rlc_map* map = nullptr;
    rlc_method* m = nullptr;
    if (rlc_map_create(occ.data(), W, H, &map) == RLC_OK) rlc_method_create(map, kind, 40.0f, td, &m);
    return m;
}

int sensor(rlc_method* m, int K) { return rlc_set_sensor_model(m, std::vector<double>((size_t)K * K, 0.5).data(), K); }

// A batch whose method gets another sensor table, trig override or none runs on what the method has now.
int batch_tables() {
    for (int kind : {RLC_RM, RLC_BL}) {
        rlc_method *a = method(kind), *b = method(kind);
        CHECK(a && b && sensor(a, 41) == RLC_OK && sensor(b, 41) == RLC_OK);
        std::vector<float> x(4000, 1.0f);
        std::vector<double> w(100);
        const rlc_filter_desc d[2] = {{a, x.data(), x.data(), x.data(), nullptr, w.data(), 50, 7},
                                      {b, x.data(), x.data(), x.data(), nullptr, w.data(), 50, 7}};
        rlc_batch* q = nullptr;
        CHECK(rlc_batch_create(d, 2, 0, &q) == RLC_OK && rlc_batch_run(q, nullptr) == RLC_OK);
        auto fresh = [&]() { return !last_graph.empty() && stale_words(last_graph.back().words[0]) == 0; };
        CHECK(fresh());
        CHECK(sensor(b, 33) == RLC_OK && rlc_batch_run(q, nullptr) == RLC_OK && fresh());
        CHECK(rlc_method_set_trig_override(a, x.data(), 350) == RLC_OK);
        CHECK(rlc_batch_run(q, nullptr) == RLC_OK && fresh());
        // every changed method is looked at, not only the first
        CHECK(sensor(a, 30) == RLC_OK && rlc_method_set_trig_override(b, x.data(), 349) == RLC_OK);
        CHECK(rlc_batch_run(q, nullptr) == RLC_ERR_ARG);
        CHECK(rlc_method_set_trig_override(b, nullptr, 0) == RLC_OK && rlc_batch_run(q, nullptr) == RLC_OK && fresh());
        // a table that could not be uploaded: refused until there is one
        refuse_from = 8 * 60 * 60;
        CHECK(sensor(a, 60) != RLC_OK);
        refuse_from = ~(size_t)0;
        CHECK(rlc_batch_run(q, nullptr) == RLC_ERR_STATE && rlc_batch_set_schedule(q, 0, 0, 256, 0) == RLC_ERR_STATE);
        CHECK(rlc_batch_run(q, nullptr) == RLC_ERR_STATE);
        CHECK(sensor(a, 60) == RLC_OK && rlc_batch_run(q, nullptr) == RLC_OK && fresh());
        rlc_batch_destroy(q);
    }
    return 0;
}

// The filter table is replaced only when no run reads it.
int batch_in_flight() {
    rlc_method* m = method(RLC_RM);
    CHECK(m && sensor(m, 41) == RLC_OK);
    std::vector<float> x(400, 1.0f);
    std::vector<double> w(50);
    const rlc_filter_desc d = {m, x.data(), x.data(), x.data(), nullptr, w.data(), 50, 7};
    rlc_batch* q = nullptr;
    CHECK(rlc_batch_create(&d, 1, 0, &q) == RLC_OK);
    for (int layout : {0, 4, 5}) CHECK(rlc_batch_run(q, nullptr) == RLC_OK && rlc_batch_set_schedule(q, layout, 0, 256, 8) == RLC_OK);
    CHECK(torn == 0);
    // the first override of a method frees nothing, which would wait for the run
    std::vector<float> trig(700, 0.5f);
    CHECK(rlc_batch_run(q, nullptr) == RLC_OK && rlc_method_set_trig_override(m, trig.data(), 350) == RLC_OK);
    CHECK(rlc_batch_run(q, nullptr) == RLC_OK && torn == 0);
    return 0;
}

size_t live_bytes() {
    size_t n = 0;
    for (const auto& b : blocks) n += b.second.live ? b.second.bytes : 0;
    return n;
}

// A Bresenham method keeps one byte a cell of free distances, and does without where there is no room.
int bresenham_memory() {
    std::vector<uint8_t> occ(300 * 200, 0);
    rlc_map* map = nullptr;
    rlc_method *m = nullptr, *late = nullptr;
    CHECK(rlc_map_create(occ.data(), 300, 200, &map) == RLC_OK);
    const size_t before = live_bytes();
    refuse_from = 300 * 200;
    CHECK(rlc_method_create(map, RLC_BL, 40.0f, 0, &m) == RLC_OK && rlc_method_destroy(m) == RLC_OK);
    CHECK(live_bytes() == before);
    refuse_from = ~(size_t)0;
    CHECK(rlc_method_create(map, RLC_BL, 40.0f, 0, &late) == RLC_OK);
    CHECK(live_bytes() >= before + 301 * 201 && live_bytes() < before + 301 * 201 + 1024);
    return 0;
}

// A map's occupancy is given without the GPU (a capture may be under way, or this be a forked child).
int occupancy() {
    for (int mode : {RLC_HOST_AUTO, RLC_HOST_STAGED}) {
        std::vector<uint8_t> occ(29 * 19, 0), got(29 * 19, 7);
        rlc_map* map = nullptr;
        on_launch = [](const std::string& name, void** args) {   // the tiles' copy into host memory
            if (name.find("k_copy_bits") != std::string::npos) memcpy(*(void**)args[2], *(void**)args[0], 8 * *(size_t*)args[1]);
        };
        CHECK(rlc_set_host_path(mode) == RLC_OK && rlc_map_create_rows(occ.data(), 29, 19, &map) == RLC_OK);
        const long long before = calls;
        CHECK(rlc_map_occupancy(map, got.data()) == RLC_OK && calls == before);
        // the stand-in's tiles are bytes of 1: of eight rows, the first is occupied
        for (int x = 0; x < 29; ++x)
            for (int y = 0; y < 19; ++y) CHECK(got[x * 19 + y] == (y % 8 == 0));
        CHECK(rlc_map_destroy(map) == RLC_OK && live_bytes() == 0);
    }
    return 0;
}

// A kernel's limit of shared memory is the device's, not the launch's: a call that lowered it could have it
// lowered between another thread's call and that one's launch.
int shared_memory_limits() {
    long long longest = 0;
    on_launch = [&](const std::string& name, void** args) {
        if (name.find("k_edges") != std::string::npos) **(uint32_t**)args[6] = 5;
        if (name.find("k_count_stats") != std::string::npos) {
            unsigned long long* out = *(unsigned long long**)args[2];
            out[0] = (unsigned long long)longest;
            out[1] = 1000;
        }
    };
    const int sides[] = {20000, 13000, 24000};
    const long long bins[] = {30000, 9000, 20000};
    for (int i = 0; i < 3; ++i) {
        longest = bins[i];
        CHECK(method(RLC_CDDT, sides[i], 8, 16));
    }
    for (int layout : {0, 3})
        for (int na : {7000, 6500, 16384, 6400}) {
            rlc_method* m = method(RLC_RM);
            std::vector<float> x(50000, 1.0f);
            double w[2];
            CHECK(m && sensor(m, 41) == RLC_OK && rlc_method_set_schedule(m, layout, 0, 0, 0) == RLC_OK);
            CHECK(rlc_calc_range_repeat_angles_eval_sensor_model(m, x.data(), x.data(), x.data(), w, 2, na, 0, nullptr) == RLC_OK);
        }
    int large = 0;
    for (const auto& k : smem_limit) large += k.second > 48 * 1024;
    CHECK(large >= 5);   // k_project_block twice, k_sort_unique, k_fused, k_bm_weights
    CHECK(lowered == 0);
    return 0;
}

// A kernel of the learned surrogate whose bounded wait runs out raises a bit and leaves its outputs
// unwritten: the call that follows it up says so, once, and the next one is good again.
int learned_timeouts() {
    const char* raises = "";    // the kernel whose wait runs out (of a training step, k_top stands for its layers)
    unsigned* word = nullptr;   // the model's error bits
    on_launch = [&](const std::string& name, void** args) {
        if (name.find("k_resolve") != std::string::npos) **(int**)args[8] = 5;
        if (name.find("k_mlp_forward") != std::string::npos) word = *(unsigned**)args[7];
        if (*raises && name.find(raises) != std::string::npos) *word |= 16u;
    };
    rlc_method* rm = method(RLC_RM);
    rlc_learned* l = nullptr;
    CHECK(rm && rlc_learned_create(rm, 1, &l) == RLC_OK);
    std::vector<float> ins(30, 1.0f), out(60), grads((size_t)rlc_learned_param_count());
    int64_t recast = 0;
    float loss = 0;
    auto query = [&]() { return rlc_learned_calc_range_repeat_angles(l, ins.data(), ins.data(), out.data(), 10, 6, nullptr, &recast, nullptr); };
    std::vector<float> xyt(128 * 3, 1.0f), t(128, 1.0f);
    auto train = [&]() { return rlc_learned_train(l, 1, 128, 1e-3f, 1, &loss, nullptr); };
    auto gradients = [&]() { return rlc_learned_gradients(l, xyt.data(), t.data(), 128, grads.data(), &loss); };
    CHECK(query() == RLC_OK && recast == 5 && train() == RLC_OK && gradients() == RLC_OK);
    raises = "k_mlp_forward";
    CHECK(query() == RLC_ERR_CUDA && std::string(rlc_last_error()).find("timed out") != std::string::npos);
    raises = "";
    CHECK(query() == RLC_OK && train() == RLC_OK && gradients() == RLC_OK);
    for (auto& call : {std::function<int()>(train), std::function<int()>(gradients)}) {
        raises = "k_top";
        CHECK(call() == RLC_ERR_CUDA);
        raises = "";
        CHECK(call() == RLC_OK && query() == RLC_OK);
    }
    // a prediction does not wait: the next call that does reports it
    raises = "k_mlp_forward";
    CHECK(rlc_learned_predict(l, xyt.data(), 128, out.data(), nullptr) == RLC_OK);
    raises = "";
    CHECK(query() == RLC_ERR_CUDA && query() == RLC_OK);
    return 0;
}

// Tuning keeps what is fastest, the call's own choice without a schedule among it; it decides for the fused
// update that it times, and the other calls go on choosing for themselves.
int autotune() {
    std::vector<float> x(9, 1.0f);   // (nothing reads the arrays)
    std::vector<double> w(9);
    const int n = 2100, na = 150;
    auto ran = [](const char* part) { return last_kernel.find(part) != std::string::npos; };
    for (int kind : {RLC_RM, RLC_CDDT, RLC_GLT, RLC_BL}) {
        rlc_method* m = method(kind, 64, 48, kind == RLC_CDDT || kind == RLC_GLT ? 16 : 0);
        CHECK(m && sensor(m, 41) == RLC_OK);
        auto fused = [&]() { return rlc_calc_range_repeat_angles_eval_sensor_model(m, x.data(), x.data(), x.data(), w.data(), n, na, RLC_DEVICE_PTRS, nullptr); };
        auto many = [&]() { return rlc_calc_range_many(m, x.data(), x.data(), n, RLC_DEVICE_PTRS, nullptr); };
        auto tune = [&](const char* fast) {
            kernel_ms = [=](const std::string& name) { return name.find(fast) != std::string::npos ? 1.0f : 2.0f; };
            return rlc_method_autotune(m, x.data(), x.data(), x.data(), w.data(), n, na, nullptr);
        };
        CHECK(many() == RLC_OK);
        const std::string own = last_kernel;
        const char* listed = kind == RLC_RM ? "k_fused<1, 1, 8>" : kind == RLC_CDDT ? "k_fused<2, 0, 2>" : "k_fused<";
        for (const char* fast : {"k_fused_wide<", listed, "k_fused_wide<"}) {
            CHECK(tune(fast) == RLC_OK && fused() == RLC_OK && ran(fast));
            CHECK(many() == RLC_OK && last_kernel == own);
            int count = 0, finals = 0, match = 0, sch[4];
            CHECK(rlc_method_autotune_results(m, 0, &count, nullptr, nullptr) == RLC_OK && count > 1);
            std::vector<int> s(4 * (size_t)count);
            std::vector<float> ms(2 * (size_t)count);
            CHECK(rlc_method_autotune_results(m, count, &count, s.data(), ms.data()) == RLC_OK);
            CHECK(rlc_method_get_schedule(m, sch, sch + 1, sch + 2, sch + 3) == RLC_OK);
            for (int i = 0; i < count; ++i)
                if (ms[2 * i + 1] > 0) {
                    ++finals;
                    match += s[4 * i] == sch[0] && s[4 * i + 2] == sch[2] && s[4 * i + 3] == sch[3];
                }
            CHECK(finals == 3 && match > 0);
        }
        // a schedule that was set holds for all calls
        CHECK(rlc_method_set_schedule(m, 0, 128, 0, 0) == RLC_OK && fused() == RLC_OK && ran("k_fused<"));
        CHECK(many() == RLC_OK && ran(kind == RLC_RM ? "k_calc_range_many<1, 0, 0" : kind == RLC_CDDT ? "k_calc_range_many<2, 0, 0" : "k_calc_range_many<"));
    }
    rlc_method* m = method(RLC_RM);
    CHECK(m && sensor(m, 41) == RLC_OK);
    const rlc_filter_desc d = {m, x.data(), x.data(), x.data(), nullptr, w.data(), 500, 70};
    rlc_batch* q = nullptr;
    CHECK(rlc_batch_create(&d, 1, 0, &q) == RLC_OK);
    auto in_graph = [&](const char* part) {
        for (const Launch& l : last_graph)
            if (l.name.find(part) != std::string::npos) return true;
        return false;
    };
    for (const char* fast : {"k_batch_wide<", "k_batch<", "k_batch_wide<"}) {
        kernel_ms = [=](const std::string& name) {
            if (name.find(fast) != std::string::npos) return 1.0f;
            return name.find("k_batch_wide<") != std::string::npos || name.find("k_batch<") != std::string::npos ? 9.0f : 0.1f;
        };
        CHECK(rlc_batch_autotune(q, nullptr) == RLC_OK && rlc_batch_run(q, nullptr) == RLC_OK && in_graph(fast));
    }
    return 0;
}

}  // namespace

int main(int argc, char** argv) {
    const std::map<std::string, int (*)()> scenarios = {{"batch_tables", batch_tables}, {"batch_in_flight", batch_in_flight},
                                                          {"bresenham_memory", bresenham_memory}, {"occupancy", occupancy},
                                                          {"shared_memory_limits", shared_memory_limits},
                                                          {"learned_timeouts", learned_timeouts}, {"autotune", autotune}};
    const auto it = scenarios.find(argc > 1 ? argv[1] : "");
    if (it == scenarios.end()) return wrong("no such scenario");
    if (const int rc = it->second()) return rc;
    printf("ok\n");
    return 0;
}
