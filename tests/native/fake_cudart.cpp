// A CUDA runtime without a GPU, for CPU tests of the library's host side: the objects of the library are linked with
// it instead of libcudart. Device memory is host memory, launches are recorded and run nothing, an allocation can
// be made to fail, and work of the default stream that nothing waited for is counted.
#include <cuda_runtime_api.h>

#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <map>
#include <set>
#include <string>
#include <vector>

namespace {
struct Launch {
    std::string name;
    int device;
    unsigned grid;
    uint64_t arg[10];  // the first eight bytes of each argument (where the kernel has as many)
};
std::map<const void*, std::string> g_names;
std::map<std::pair<const void*, int>, int> g_smem;  // dynamic shared memory limit, by kernel and device
std::vector<Launch> g_launches;
std::vector<float> g_elapsed;
std::set<void*> g_live;
size_t g_next_elapsed = 0;
int g_fail = 0, g_device = 0, g_pending = 0, g_streams = 0;
cudaError_t g_last = cudaSuccess;
struct Config {
    dim3 grid, block;
    size_t smem;
    cudaStream_t stream;
};
std::vector<Config> g_config;

int args_of(const std::string& n) {
    auto has = [&](const char* s) { return n.find(s) != std::string::npos; };
    if (has("k_step_tiled") || has("k_tile_masks")) return 9;
    if (has("k_sweep_tiled") || has("k_step_ensemble")) return 7;
    return 0;
}
cudaError_t launch(const void* f, dim3 grid, size_t smem, cudaStream_t st, void** args) {
    Launch l{};
    l.name = g_names.count(f) ? g_names[f] : "?";
    l.device = g_device;
    l.grid = grid.x;
    for (int i = 0; i < args_of(l.name); ++i) {
        const bool wide = !(l.name.find("k_tile_masks") != std::string::npos && i >= 2 && i <= 7 && i != 6) &&
                          !(l.name.find("k_step_ensemble") != std::string::npos && i == 4);
        std::memcpy(&l.arg[i], args[i], wide ? 8 : 4);
    }
    if (smem > 48 * 1024 && g_smem[{f, g_device}] < (int)smem) return g_last = cudaErrorInvalidValue;
    if (!st) ++g_pending;
    g_launches.push_back(l);
    return cudaSuccess;
}
}  // namespace

extern "C" {

// ---- what the tests use
void fk_reset() {
    g_launches.clear();
    g_elapsed.clear();
    g_next_elapsed = 0;
    g_fail = g_pending = g_device = 0;
    g_last = cudaSuccess;
}
void fk_fail_malloc(int n) { g_fail = n; }  // the n-th allocation from now fails (0: none)
int fk_pending() { return g_pending; }      // default-stream operations that nothing has waited for
int fk_live() { return (int)g_live.size(); }
int fk_is_live(void* p) { return (int)g_live.count(p); }
int fk_launches() { return (int)g_launches.size(); }
const char* fk_name(int i) { return g_launches[i].name.c_str(); }
unsigned fk_grid(int i) { return g_launches[i].grid; }
int fk_device(int i) { return g_launches[i].device; }
uint64_t fk_arg(int i, int a) { return g_launches[i].arg[a]; }
void fk_elapsed(const float* ms, int n) { g_elapsed.assign(ms, ms + n); }
void fk_set_device(int d) { g_device = d; }

// ---- registration and launches
void** __cudaRegisterFatBinary(void*) {
    static void* h;
    return &h;
}
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterFunction(void**, const char* host, char*, const char* name, int, void*, void*, void*, void*, int*) {
    g_names[host] = name;
}
void __cudaRegisterVar(void**, char*, char*, const char*, int, size_t, int, int) {}
unsigned __cudaPushCallConfiguration(dim3 g, dim3 b, size_t smem, cudaStream_t st) {
    g_config.push_back(Config{g, b, smem, st});
    return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3* g, dim3* b, size_t* smem, void* st) {
    const Config c = g_config.back();
    g_config.pop_back();
    *g = c.grid, *b = c.block, *smem = c.smem, *(cudaStream_t*)st = c.stream;
    return cudaSuccess;
}
cudaError_t cudaLaunchKernel(const void* f, dim3 grid, dim3, void** args, size_t smem, cudaStream_t st) {
    return launch(f, grid, smem, st, args);
}
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t* c, const void* f, void** args) {
    return launch(f, c->gridDim, c->dynamicSmemBytes, c->stream, args);
}
cudaError_t cudaFuncSetAttribute(const void* f, cudaFuncAttribute a, int v) {
    if (a == cudaFuncAttributeMaxDynamicSharedMemorySize) g_smem[{f, g_device}] = v;
    return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int* n, const void*, int, size_t, unsigned) {
    *n = 4;
    return cudaSuccess;
}

// ---- memory
cudaError_t cudaMalloc(void** p, size_t n) {
    if (g_fail > 0 && --g_fail == 0) {
        *p = nullptr;
        return g_last = cudaErrorMemoryAllocation;
    }
    *p = std::malloc(n ? n : 1);
    std::memset(*p, 0xA5, n);
    g_live.insert(*p);
    return cudaSuccess;
}
cudaError_t cudaFree(void* p) {
    if (!p) return cudaSuccess;
    if (!g_live.erase(p)) {
        std::fprintf(stderr, "fake runtime: cudaFree of an unknown pointer\n");
        std::abort();
    }
    std::free(p);
    return cudaSuccess;
}
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind k) {
    std::memcpy(d, s, n);
    if (k != cudaMemcpyDeviceToHost) ++g_pending;  // pageable memory: the last part may still be on its way
    return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t st) {
    std::memcpy(d, s, n);
    if (!st) ++g_pending;
    return cudaSuccess;
}
cudaError_t cudaMemset(void* d, int v, size_t n) { return cudaMemsetAsync(d, v, n, nullptr); }
cudaError_t cudaMemsetAsync(void* d, int v, size_t n, cudaStream_t st) {
    std::memset(d, v, n);
    if (!st) ++g_pending;
    return cudaSuccess;
}

// ---- streams, events, graphs, devices
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* st, unsigned) {
    *st = (cudaStream_t)(uintptr_t)(0x1000 + 16 * ++g_streams);
    return cudaSuccess;
}
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t st) {
    if (!st) g_pending = 0;
    return cudaSuccess;
}
cudaError_t cudaStreamGetDevice(cudaStream_t, int* d) {
    *d = g_device;
    return cudaSuccess;
}
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) { return cudaSuccess; }
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t* g) {
    *g = (cudaGraph_t)(uintptr_t)0x10;
    return cudaSuccess;
}
cudaError_t cudaGraphInstantiate(cudaGraphExec_t* e, cudaGraph_t, unsigned long long) {
    *e = (cudaGraphExec_t)(uintptr_t)0x20;
    return cudaSuccess;
}
cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaGraphUpload(cudaGraphExec_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t* e) {
    *e = (cudaEvent_t)(uintptr_t)0x30;
    return cudaSuccess;
}
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) {
    *ms = g_next_elapsed < g_elapsed.size() ? g_elapsed[g_next_elapsed++] : 1.0f;
    return cudaSuccess;
}
cudaError_t cudaGetDevice(int* d) {
    *d = g_device;
    return cudaSuccess;
}
cudaError_t cudaSetDevice(int d) {
    g_device = d;
    return cudaSuccess;
}
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr, int) {
    *v = 148;
    return cudaSuccess;
}
cudaError_t cudaGetLastError() {
    const cudaError_t e = g_last;
    g_last = cudaSuccess;
    return e;
}
const char* cudaGetErrorString(cudaError_t e) { return e == cudaSuccess ? "no error" : "fake error"; }
cudaError_t cudaGetSymbolAddress(void** p, const void*) {
    static int word;
    *p = &word;
    return cudaSuccess;
}
// the one driver entry that the library asks for is cuTensorMapEncodeTiled
static int encode_tiled(void* map, int, unsigned, void* base, ...) {
    std::memcpy(map, &base, sizeof(base));
    return 0;
}
cudaError_t cudaGetDriverEntryPoint(const char*, void** f, unsigned long long, cudaDriverEntryPointQueryResult* q) {
    *f = (void*)encode_tiled;
    if (q) *q = cudaDriverEntryPointSuccess;
    return cudaSuccess;
}

}  // extern "C"
