// A stand-in for the CUDA runtime on a machine without a GPU, which keeps the books of what a call may rely on: device
// memory is host memory, kernels do nothing, and every upload or clearing of device memory counts as outstanding on its
// stream until the host waits for that stream. A launch on a stream that is not ordered behind an outstanding one (a
// non-blocking stream and any other) is recorded. A pageable cudaMemcpy counts as outstanding too: it may return once
// the source has been staged. The first kernel launched since fake_forget() is kept, to tell the routes of calls apart.
#include <cstddef>
#include <cstdint>
#include <cstdlib>
#include <cstring>
#include <map>
#include <string>

namespace {
struct Dim3 {
    unsigned x, y, z;
};
struct Stream {
    bool nonblocking;
    int outstanding;
};
std::map<void*, Stream> g_streams;
std::map<void*, size_t> g_pinned;
std::string g_unordered;
size_t g_host_limit = ~size_t(0);
int g_launches = 0, g_first_block = 0;
const void* g_first_kernel = nullptr;
struct Config {
    Dim3 grid, block;
    size_t smem;
    void* stream;
} g_config;

Stream& stream(void* s) {
    if (s == reinterpret_cast<void*>(1)) s = nullptr;
    return g_streams[s];
}
void wait_for(void* s) {
    stream(s).outstanding = 0;
    if (s == nullptr)
        for (auto& e : g_streams)
            if (!e.second.nonblocking) e.second.outstanding = 0;
}
void wait_all() {
    for (auto& e : g_streams) e.second.outstanding = 0;
}
void queued(void* s) { ++stream(s).outstanding; }
bool pinned(const void* p) {
    for (const auto& e : g_pinned)
        if (p >= e.first && p < static_cast<char*>(e.first) + e.second) return true;
    return false;
}
int launch(const void* kernel, Dim3 block, void* s) {
    if (g_launches++ == 0) g_first_kernel = kernel, g_first_block = static_cast<int>(block.x);
    stream(s);
    for (const auto& e : g_streams) {
        if (e.first == s || e.second.outstanding == 0) continue;
        const bool ordered = (s == nullptr && !e.second.nonblocking) || (e.first == nullptr && !stream(s).nonblocking);
        if (!ordered)
            g_unordered += "launch " + std::to_string(g_launches) + " beside " +
                           std::to_string(e.second.outstanding) + " outstanding on another stream; ";
    }
    if (s == nullptr) queued(s);  // (a later launch on a non-blocking stream does not wait for it)
    return 0;
}
}  // namespace

extern "C" {
const char* fake_unordered() { return g_unordered.c_str(); }
int fake_launches() { return g_launches; }
const void* fake_first_kernel() { return g_first_kernel; }
int fake_first_block() { return g_first_block; }
void fake_forget() { g_unordered.clear(), g_launches = 0; }
int fake_outstanding() {
    int n = 0;
    for (const auto& e : g_streams) n += e.second.outstanding;
    return n;
}
void fake_host_limit(size_t bytes) { g_host_limit = bytes; }
size_t fake_pinned_bytes() {
    size_t n = 0;
    for (const auto& e : g_pinned) n += e.second;
    return n;
}

int cudaGetDeviceCount(int* n) { return *n = 1, 0; }
int cudaGetDevice(int* d) { return *d = 0, 0; }
int cudaSetDevice(int) { return 0; }
int cudaDeviceGetAttribute(int* v, int attr, int) { return *v = attr == 16 ? 148 : attr == 97 ? 232448 : 1, 0; }
int cudaGetDeviceProperties_v2(void*, int) { return 0; }
int cudaDeviceSynchronize() { return wait_all(), 0; }
const char* cudaGetErrorString(int) { return "fake"; }
int cudaGetLastError() { return 0; }
int cudaMemGetInfo(size_t* f, size_t* t) { return *f = *t = size_t(100) << 30, 0; }

int cudaMalloc(void** p, size_t n) { return (*p = std::calloc(n, 1)) ? 0 : 2; }
int cudaFree(void* p) { return wait_all(), std::free(p), 0; }
int cudaHostAlloc(void** p, size_t n, unsigned) {
    if (n > g_host_limit) return 2;
    *p = std::aligned_alloc(4096, (n + 4095) / 4096 * 4096);
    std::memset(*p, 0, n);
    g_pinned[*p] = n;
    return 0;
}
int cudaFreeHost(void* p) { return g_pinned.erase(p), std::free(p), 0; }
int cudaHostGetDevicePointer(void** d, void* h, unsigned) { return *d = h, 0; }
int cudaGetSymbolAddress(void** p, const void*) {
    static char symbol[1 << 20];
    return *p = symbol, 0;
}

int cudaMemcpy(void* d, const void* s, size_t n, int kind) {
    std::memcpy(d, s, n);
    if (kind == 1 && !pinned(s)) queued(nullptr);
    else wait_for(nullptr);
    return 0;
}
int cudaMemcpyAsync(void* d, const void* s, size_t n, int kind, void* st) {
    std::memcpy(d, s, n);
    if (kind == 1) queued(st);
    return 0;
}
int cudaMemset(void* d, int v, size_t n) { return std::memset(d, v, n), queued(nullptr), 0; }
int cudaMemsetAsync(void* d, int v, size_t n, void* st) { return std::memset(d, v, n), queued(st), 0; }

int cudaStreamCreateWithFlags(void** s, unsigned flags) {
    *s = std::malloc(16);
    g_streams[*s] = {(flags & 1u) != 0, 0};
    return 0;
}
int cudaStreamDestroy(void* s) { return g_streams.erase(s), std::free(s), 0; }
int cudaStreamSynchronize(void* s) { return wait_for(s), 0; }
int cudaStreamWaitEvent(void*, void*, unsigned) { return 0; }
int cudaStreamBeginCapture(void*, int) { return 0; }
int cudaStreamEndCapture(void*, void** g) { return *g = nullptr, 0; }
int cudaGraphInstantiate(void** e, void*, unsigned long long) { return *e = nullptr, 0; }
int cudaGraphLaunch(void*, void*) { return 0; }
int cudaGraphDestroy(void*) { return 0; }
int cudaGraphExecDestroy(void*) { return 0; }
int cudaEventCreate(void** e) { return *e = std::malloc(16), 0; }
int cudaEventCreateWithFlags(void** e, unsigned) { return *e = std::malloc(16), 0; }
int cudaEventDestroy(void* e) { return std::free(e), 0; }
int cudaEventRecord(void*, void*) { return 0; }
int cudaEventSynchronize(void*) { return 0; }
int cudaEventElapsedTime(float* ms, void*, void*) { return *ms = 0.0f, 0; }

int cudaFuncSetAttribute(const void*, int, int) { return 0; }
int cudaOccupancyMaxActiveBlocksPerMultiprocessor(int* n, const void*, int, size_t) { return *n = 1, 0; }
int cudaLaunchKernel(const void* f, Dim3, Dim3 b, void**, size_t, void* s) { return launch(f, b, s); }
int cudaLaunchCooperativeKernel(const void* f, Dim3, Dim3 b, void**, size_t, void* s) { return launch(f, b, s); }
int cudaLaunchKernelExC(const Config* c, const void* f, void**) { return launch(f, c->block, c->stream); }

unsigned __cudaPushCallConfiguration(Dim3 grid, Dim3 block, size_t smem, void* s) {
    return g_config = {grid, block, smem, s}, 0u;
}
int __cudaPopCallConfiguration(Dim3* grid, Dim3* block, size_t* smem, void* s) {
    *grid = g_config.grid, *block = g_config.block, *smem = g_config.smem;
    std::memcpy(s, &g_config.stream, sizeof(void*));
    return 0;
}
void** __cudaRegisterFatBinary(void*) {
    static void* handle[4];
    return handle;
}
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterFunction(void**, const char*, char*, const char*, int, void*, void*, void*, void*, int*) {}
void __cudaRegisterVar(void**, char*, char*, const char*, int, size_t, int, int) {}
}
