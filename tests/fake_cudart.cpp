// A CUDA runtime without a GPU, for tests of the library's host code.
//
// Device memory is host memory and kernels do nothing, so what the host code
// hands to the runtime can be checked: uploads that another stream does not
// wait for, launches with a null or freed pointer, stream waits, and the code
// after a failed allocation.
#include <cuda_runtime_api.h>
#include <cxxabi.h>

#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <map>
#include <string>
#include <vector>

namespace {

std::map<uintptr_t, size_t> live, freed;      // device and pinned memory
std::map<const void *, std::string> kernels;  // host function -> demangled name
std::string events;                           // one line per launch, wait and fault
long allocations = 0, fail_at = -1, faults = 0, live_streams = 0;
int pending = 0;     // legacy-stream copies and fills that nothing has waited for
int refine_script = 0;   // refine_classify_kernel: 0 accepts every block, 1 finds one cluster in each
cudaError_t last = cudaSuccess;

struct Stream {
    unsigned long long id;
    bool capturing;
};
std::vector<Stream *> spare;   // destroyed streams: their handles are given out again
unsigned long long next_id = 10;

void fault(const std::string &what) {
    faults++;
    events += "FAULT " + what + "\n";
}
bool inside(const std::map<uintptr_t, size_t> &m, const void *p) {
    auto it = m.upper_bound((uintptr_t)p);
    if (it == m.begin()) return false;
    --it;
    return (uintptr_t)p < it->first + it->second;
}
cudaError_t allocate(void **p, size_t n) {
    if (allocations++ == fail_at) {
        *p = nullptr;
        return cudaErrorMemoryAllocation;
    }
    *p = calloc(n, 1);
    live[(uintptr_t)*p] = n;
    return cudaSuccess;
}
cudaError_t release(void *p) {
    if (!p) return cudaSuccess;
    auto it = live.find((uintptr_t)p);
    if (it == live.end()) {
        fault("free of memory that is not allocated");
        return cudaErrorInvalidValue;
    }
    freed[it->first] = it->second;   // never handed out again: a later use shows
    live.erase(it);
    pending = 0;   // a free waits for the device
    return cudaSuccess;
}
bool legacy(cudaStream_t s) { return s == nullptr || s == cudaStreamLegacy; }
// work on a stream that the legacy stream is not ordered with
void on_stream(cudaStream_t s, const std::string &what) {
    if (!legacy(s) && pending) fault("an upload may still be running at " + what);
}
// the parameter types of a demangled function
std::vector<std::string> parameters(const std::string &f) {
    std::vector<std::string> out;
    int angle = 0, paren = 0;
    std::string cur;
    for (char c : f) {
        if (c == '<') angle++;
        if (c == '>') angle--;
        if (c == '(' && angle == 0 && paren++ == 0) continue;
        if (c == ')' && angle == 0 && --paren == 0) break;
        if (paren == 0) continue;
        if (c == ',' && angle == 0 && paren == 1) {
            out.push_back(cur);
            cur.clear();
        } else {
            cur += c;
        }
    }
    if (!cur.empty()) out.push_back(cur);
    return out;
}
cudaError_t launch(const void *f, dim3 grid, void **args, cudaStream_t s) {
    const std::string &name = kernels[f];
    on_stream(s, name.substr(0, name.find('(')));
    std::string mask;
    const auto par = parameters(name);
    for (size_t k = 0; k < par.size(); k++) {
        if (par[k].back() != '*') continue;
        const void *p = *(void **)args[k];
        if (inside(freed, p) && !inside(live, p)) fault("freed memory given to " + name);
        mask += p ? 'x' : '0';
    }
    events += "launch " + name.substr(0, name.find('(')) + " " + mask + "\n";
    if (name.find("refine_classify_kernel") != std::string::npos) {
        int *bstate = *(int **)args[3], *state = *(int **)args[12], *nbad = *(int **)args[13], *nedge = *(int **)args[14];
        int2 *edges = *(int2 **)args[15];
        const size_t cap = 32768;   // kRefineEdgeCap
        for (unsigned b = 0; b < grid.x; b++) {
            if (bstate[b] != 0 && bstate[b] != 3) continue;
            state[b] = refine_script && bstate[b] == 0 ? 0 : 1;
            nbad[b] = nedge[b] = state[b] == 0;
            if (state[b] == 0) edges[b * cap] = int2{0, 1};
            bstate[b] = state[b];
        }
    }
    return cudaSuccess;
}

}  // namespace

extern "C" {

// ------------------------------------------------ for the tests
void fake_fail_at(long k) {   // the k-th allocation from now fails (-1: none)
    allocations = 0;
    fail_at = k;
}
long fake_allocations() { return allocations; }
long fake_faults() { return faults; }
long fake_live() { return (long)live.size() + live_streams; }
const char *fake_events() { return events.c_str(); }
void fake_clear() {
    events.clear();
    faults = 0;
}
void fake_refine_script(int k) { refine_script = k; }
void fake_capture(cudaStream_t s, int on) { ((Stream *)s)->capturing = on; }

// ------------------------------------------------ memory
cudaError_t cudaMalloc(void **p, size_t n) { return allocate(p, n); }
cudaError_t cudaHostAlloc(void **p, size_t n, unsigned) { return allocate(p, n); }
cudaError_t cudaMallocHost(void **p, size_t n) { return allocate(p, n); }
cudaError_t cudaFree(void *p) { return release(p); }
cudaError_t cudaFreeHost(void *p) { return release(p); }
cudaError_t cudaHostGetDevicePointer(void **d, void *h, unsigned) {
    *d = h;
    return cudaSuccess;
}
cudaError_t cudaMemcpy(void *d, const void *s, size_t n, cudaMemcpyKind kind) {
    if (!d || !s) return cudaErrorInvalidValue;
    memcpy(d, s, n);
    pending = kind == cudaMemcpyHostToDevice ? pending + 1 : 0;
    return cudaSuccess;
}
cudaError_t cudaMemset(void *d, int v, size_t n) {
    if (!d) return cudaErrorInvalidValue;
    memset(d, v, n);
    pending++;
    return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, cudaMemcpyKind, cudaStream_t st) {
    if (n && (!d || !s)) return cudaErrorInvalidValue;
    on_stream(st, "cudaMemcpyAsync");
    memcpy(d, s, n);
    return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void *d, int v, size_t n, cudaStream_t st) {
    if (n && !d) return cudaErrorInvalidValue;
    on_stream(st, "cudaMemsetAsync");
    memset(d, v, n);
    return cudaSuccess;
}

// ------------------------------------------------ streams and events
cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned) {
    Stream *p = spare.empty() ? new Stream : spare.back();
    if (!spare.empty()) spare.pop_back();
    *p = Stream{next_id++, false};
    *s = (cudaStream_t)p;
    live_streams++;
    return cudaSuccess;
}
cudaError_t cudaStreamDestroy(cudaStream_t s) {
    spare.push_back((Stream *)s);
    live_streams--;
    return cudaSuccess;
}
cudaError_t cudaStreamGetId(cudaStream_t s, unsigned long long *id) {
    if (!legacy(s) && ((Stream *)s)->capturing) return cudaErrorStreamCaptureUnsupported;
    *id = legacy(s) ? 1 : ((Stream *)s)->id;
    return cudaSuccess;
}
cudaError_t cudaStreamIsCapturing(cudaStream_t s, cudaStreamCaptureStatus *st) {
    *st = !legacy(s) && ((Stream *)s)->capturing ? cudaStreamCaptureStatusActive : cudaStreamCaptureStatusNone;
    return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t s) {
    if (legacy(s)) pending = 0;
    events += "synchronize\n";
    return cudaSuccess;
}
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) {
    events += "wait\n";
    return cudaSuccess;
}
cudaError_t cudaDeviceSynchronize() {
    pending = 0;
    return cudaSuccess;
}
cudaError_t cudaEventCreate(cudaEvent_t *e) {
    *e = (cudaEvent_t)malloc(1);
    return cudaSuccess;
}
cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned) { return cudaEventCreate(e); }
cudaError_t cudaEventDestroy(cudaEvent_t e) {
    free(e);
    return cudaSuccess;
}
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float *ms, cudaEvent_t, cudaEvent_t) {
    *ms = 1.0f;
    return cudaSuccess;
}

// ------------------------------------------------ device and launches
cudaError_t cudaGetDevice(int *d) {
    *d = 0;
    return cudaSuccess;
}
cudaError_t cudaGetDeviceCount(int *n) {
    *n = 1;
    return cudaSuccess;
}
cudaError_t cudaDeviceGetAttribute(int *v, cudaDeviceAttr, int) {
    *v = 148;
    return cudaSuccess;
}
cudaError_t cudaFuncGetAttributes(cudaFuncAttributes *a, const void *) {
    memset(a, 0, sizeof *a);
    return cudaSuccess;
}
cudaError_t cudaFuncSetAttribute(const void *, cudaFuncAttribute, int) { return cudaSuccess; }
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int *n, const void *, int, size_t, unsigned) {
    *n = 2;
    return cudaSuccess;
}
cudaError_t cudaGetLastError() { return last; }
const char *cudaGetErrorString(cudaError_t e) { return e == cudaErrorMemoryAllocation ? "out of memory" : "error"; }
cudaError_t cudaGetDriverEntryPoint(const char *, void **, unsigned long long, cudaDriverEntryPointQueryResult *r) {
    *r = cudaDriverEntryPointSymbolNotFound;
    return cudaErrorNotSupported;
}
cudaError_t cudaGetSymbolAddress(void **p, const void *) {
    *p = nullptr;
    return cudaErrorInvalidSymbol;
}
cudaError_t cudaLaunchKernel(const void *f, dim3 grid, dim3, void **args, size_t, cudaStream_t s) {
    return launch(f, grid, args, s);
}
cudaError_t cudaLaunchCooperativeKernel(const void *f, dim3 grid, dim3, void **args, size_t, cudaStream_t s) {
    return launch(f, grid, args, s);
}

// ------------------------------------------------ what nvcc's host code calls
static struct {
    dim3 grid, block;
    size_t smem;
    void *stream;
} config;
unsigned __cudaPushCallConfiguration(dim3 grid, dim3 block, size_t smem, void *stream) {
    config.grid = grid;
    config.block = block;
    config.smem = smem;
    config.stream = stream;
    return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3 *grid, dim3 *block, size_t *smem, void *stream) {
    *grid = config.grid;
    *block = config.block;
    *smem = config.smem;
    *(void **)stream = config.stream;
    return cudaSuccess;
}
void **__cudaRegisterFatBinary(void *) {
    static void *handle;
    return &handle;
}
void __cudaRegisterFatBinaryEnd(void **) {}
void __cudaUnregisterFatBinary(void **) {}
void __cudaRegisterFunction(void **, const char *host, char *, const char *name, int, void *, void *, void *, void *,
                            int *) {
    int st = 0;
    char *d = abi::__cxa_demangle(name, nullptr, nullptr, &st);
    std::string s = st == 0 ? d : name;
    free(d);
    if (s.rfind("void ", 0) == 0) s = s.substr(5);
    kernels[host] = s;
}
void __cudaRegisterVar(void **, char *, char *, const char *, int, size_t, int, int) {}

}  // extern "C"
