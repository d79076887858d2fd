// A CUDA runtime for the CPU tests: the library's objects link against it
// instead of libcudart, so that the host runtime's bookkeeping runs without a
// GPU. Device memory is host memory; every copy, and every buffer that a
// launch of the marker scheduler, the forcing pass or the step names, is held
// against the allocations (fake_checks.cu). Kernels do nothing. A test can let an allocation fail, set a stream under
// capture, and ask how the launches are ordered (fake_* below).
#include <cuda_runtime_api.h>
#include <cxxabi.h>

#include <algorithm>
#include <cstdlib>
#include <cstring>
#include <map>
#include <mutex>
#include <string>
#include <vector>


struct CUstream_st {
    std::map<CUstream_st*, long long> clock;   // of every stream: its last operation this stream is ordered after
};
struct CUevent_st {
    std::map<CUstream_st*, long long> clock;
};

extern "C" void fake_check(const char* name, void** args);   // fake_checks.cu

namespace {

struct Launch {
    std::string name;
    CUstream_st* stream;
    std::map<CUstream_st*, long long> after;
};

std::recursive_mutex mu;
std::map<char*, size_t> device, pinned, registered;   // (registered: the test's own pinned memory)
std::map<const void*, std::string>& names() {   // filled by static constructors
    static std::map<const void*, std::string> m;
    return m;
}
std::vector<Launch> launches;
std::string faults;
long long mallocs = 0, waits = 0, fail_in = 0;
bool capturing = false;
cudaError_t last = cudaSuccess;
struct Config {
    dim3 grid, block;
    size_t smem;
    cudaStream_t st;
} config;

cudaError_t ret(cudaError_t e) {
    if (e != cudaSuccess) last = e;
    return e;
}
void fault(const std::string& what) { faults += what + "\n"; }
bool inside(const std::map<char*, size_t>& m, const void* p, size_t n) {
    auto it = m.upper_bound((char*)p);
    if (it == m.begin()) return false;
    --it;
    return (char*)p >= it->first && (char*)p + n <= it->first + it->second;
}
// a launch or a copy uses n bytes of device memory from p
void need(const char* who, const char* what, const void* p, long long n) {
    if (n > 0 && !inside(device, p, (size_t)n))
        fault(std::string(who) + ": " + what + " does not hold " + std::to_string(n) + " bytes");
}
void not_in_capture(const char* what) {
    if (capturing) fault(std::string(what) + " under capture");
}
void order(cudaStream_t s) {
    if (s) s->clock[s]++;
}
cudaError_t allocate(std::map<char*, size_t>& where, void** p, size_t n) {
    std::lock_guard<std::recursive_mutex> lk(mu);
    not_in_capture("an allocation");
    mallocs++;
    *p = nullptr;
    if (fail_in > 0 && --fail_in == 0) return ret(cudaErrorMemoryAllocation);
    void* q = nullptr;
    if (posix_memalign(&q, 256, std::max<size_t>(n, 1))) return ret(cudaErrorMemoryAllocation);
    if (n <= (16u << 20)) std::memset(q, 0, n);
    where[(char*)q] = n;
    *p = q;
    return cudaSuccess;
}
cudaError_t release(std::map<char*, size_t>& where, void* p) {
    std::lock_guard<std::recursive_mutex> lk(mu);
    if (!p) return cudaSuccess;
    not_in_capture("a free");
    if (!where.erase((char*)p)) fault("free of an unknown pointer");
    else std::free(p);
    return cudaSuccess;
}
cudaError_t copy(void* dst, const void* src, size_t n, cudaMemcpyKind kind, cudaStream_t st) {
    std::lock_guard<std::recursive_mutex> lk(mu);
    const bool to = kind == cudaMemcpyHostToDevice || kind == cudaMemcpyDeviceToDevice;
    const bool from = kind == cudaMemcpyDeviceToHost || kind == cudaMemcpyDeviceToDevice || kind == cudaMemcpyDefault;
    const std::string before = faults;
    if (to) need("copy", "the destination", dst, (long long)n);
    if (from) need("copy", "the source", src, (long long)n);
    order(st);
    if (faults == before) std::memmove(dst, src, n);
    return cudaSuccess;
}

cudaError_t launch(const void* fn, void** args, cudaStream_t st) {
    std::lock_guard<std::recursive_mutex> lk(mu);
    const std::string& name = names()[fn];
    fake_check(name.c_str(), args);
    launches.push_back(Launch{name, st, st ? st->clock : std::map<CUstream_st*, long long>{}});
    order(st);
    return cudaSuccess;
}

}  // namespace

// for fake_checks.cu
void fake_need(const char* who, const char* what, const void* p, long long n) { need(who, what, p, n); }
void fake_fault(const char* who, const char* what) { fault(std::string(who) + ": " + what); }
bool fake_writable(const void* p, long long n) { return inside(pinned, p, (size_t)n) || inside(registered, p, (size_t)n) || inside(device, p, (size_t)n); }
bool fake_sound() { return faults.empty(); }

extern "C" {

// ---- for the tests ----
void fake_reset() {
    std::lock_guard<std::recursive_mutex> lk(mu);
    launches.clear();
    registered.clear();
    faults.clear();
    mallocs = waits = fail_in = 0;
    capturing = false;
    last = cudaSuccess;
}
void fake_fail(long long nth) { fail_in = nth; }   // the nth allocation from here fails
void fake_capture(int on) { capturing = on != 0; }
void fake_pin(void* p, size_t n) { registered[(char*)p] = n; }
long long fake_mallocs() { return mallocs; }
long long fake_waits() { return waits; }
const char* fake_faults() { return faults.c_str(); }
// an operation that is not the library's on stream s; its number
long long fake_foreign(void* s) {
    order((cudaStream_t)s);
    return ((cudaStream_t)s)->clock[(cudaStream_t)s];
}
// launches whose kernel's name holds `part`; the ones not ordered after operation `number` of stream s
long long fake_launches(const char* part) {
    return std::count_if(launches.begin(), launches.end(), [&](const Launch& l) { return l.name.find(part) != std::string::npos; });
}
long long fake_unordered(const char* part, void* s, long long number) {
    return std::count_if(launches.begin(), launches.end(), [&](Launch& l) {
        return l.name.find(part) != std::string::npos && l.after[(cudaStream_t)s] < number;
    });
}

// ---- the runtime ----
void** __cudaRegisterFatBinary(void*) { static void* h; return &h; }
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterFunction(void**, const char* host, char*, const char* name, int, uint3*, uint3*, dim3*, dim3*, int*) {
    int s = 0;
    char* d = abi::__cxa_demangle(name, nullptr, nullptr, &s);
    names()[host] = d ? d : name;
    std::free(d);
}
void __cudaRegisterVar(void**, char*, char*, const char*, int, size_t, int, int) {}
unsigned __cudaPushCallConfiguration(dim3 g, dim3 b, size_t smem, cudaStream_t st) {
    config = Config{g, b, smem, st};
    return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3* g, dim3* b, size_t* smem, void* st) {
    *g = config.grid;
    *b = config.block;
    *smem = config.smem;
    *(cudaStream_t*)st = config.st;
    return cudaSuccess;
}
cudaError_t cudaLaunchKernel(const void* fn, dim3, dim3, void** args, size_t, cudaStream_t st) { return launch(fn, args, st); }
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t* c, const void* fn, void** args) { return launch(fn, args, c->stream); }
cudaError_t cudaMalloc(void** p, size_t n) { return allocate(device, p, n); }
cudaError_t cudaFree(void* p) { return release(device, p); }
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) { return allocate(pinned, p, n); }
cudaError_t cudaFreeHost(void* p) { return release(pinned, p); }
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind k) {
    not_in_capture("cudaMemcpy");
    return copy(d, s, n, k, nullptr);
}
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind k, cudaStream_t st) { return copy(d, s, n, k, st); }
cudaError_t cudaMemcpy2DAsync(void* d, size_t dp, const void* s, size_t sp, size_t w, size_t h, cudaMemcpyKind k, cudaStream_t st) {
    for (size_t r = 0; r < h; r++) copy((char*)d + r * dp, (const char*)s + r * sp, w, k, st);
    return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void* p, int v, size_t n, cudaStream_t st) {
    std::lock_guard<std::recursive_mutex> lk(mu);
    need("memset", "the destination", p, (long long)n);
    if (n <= (16u << 20) && inside(device, p, n)) std::memset(p, v, n);   // (larger ones are the lattice's, which nothing here reads)
    order(st);
    return cudaSuccess;
}
cudaError_t cudaGetLastError() {
    const cudaError_t e = last;
    last = cudaSuccess;
    return e;
}
const char* cudaGetErrorString(cudaError_t) { return "an error of the test's"; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaGetDevice(int* d) { *d = 0; return cudaSuccess; }
cudaError_t cudaGetDeviceCount(int* n) { *n = 1; return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr a, int) {
    *v = a == cudaDevAttrComputeCapabilityMajor ? 10 : a == cudaDevAttrMultiProcessorCount ? 148 : 0;
    return cudaSuccess;
}
cudaError_t cudaDeviceGetStreamPriorityRange(int* lo, int* hi) { *lo = 0; *hi = -5; return cudaSuccess; }
cudaError_t cudaDeviceSynchronize() { return cudaSuccess; }
cudaError_t cudaMemGetInfo(size_t* f, size_t* t) { *f = *t = (size_t)180 << 30; return cudaSuccess; }
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int* n, const void*, int, size_t, unsigned) { *n = 4; return cudaSuccess; }
cudaError_t cudaFuncSetAttribute(const void*, cudaFuncAttribute, int) { return cudaSuccess; }
cudaError_t cudaStreamCreateWithPriority(cudaStream_t* s, unsigned, int) { *s = new CUstream_st(); return cudaSuccess; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) { *s = new CUstream_st(); return cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t s) { delete s; return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) {
    not_in_capture("cudaStreamSynchronize");
    waits++;
    return cudaSuccess;
}
cudaError_t cudaStreamWaitEvent(cudaStream_t s, cudaEvent_t e, unsigned) {
    for (const auto& c : e->clock) s->clock[c.first] = std::max(s->clock[c.first], c.second);
    return cudaSuccess;
}
cudaError_t cudaStreamIsCapturing(cudaStream_t, cudaStreamCaptureStatus* c) {
    *c = capturing ? cudaStreamCaptureStatusActive : cudaStreamCaptureStatusNone;
    return cudaSuccess;
}
cudaError_t cudaEventCreate(cudaEvent_t* e) { *e = new CUevent_st(); return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { return cudaEventCreate(e); }
cudaError_t cudaEventDestroy(cudaEvent_t e) { delete e; return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s) { e->clock = s->clock; return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { not_in_capture("cudaEventSynchronize"); return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) { *ms = 0.f; return cudaSuccess; }
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes* a, const void* p) {
    *a = cudaPointerAttributes{};
    a->type = inside(pinned, p, 1) || inside(registered, p, 1) ? cudaMemoryTypeHost : inside(device, p, 1) ? cudaMemoryTypeDevice : cudaMemoryTypeUnregistered;
    a->devicePointer = a->type == cudaMemoryTypeUnregistered ? nullptr : const_cast<void*>(p);
    return cudaSuccess;
}
cudaError_t cudaGetSymbolAddress(void** p, const void*) { static double scratch[8192]; *p = scratch; return cudaSuccess; }
// graphs: none here
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) { return cudaErrorNotSupported; }
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t*) { return cudaErrorNotSupported; }
cudaError_t cudaGraphGetNodes(cudaGraph_t, cudaGraphNode_t*, size_t*) { return cudaErrorNotSupported; }
cudaError_t cudaGraphNodeGetType(cudaGraphNode_t, cudaGraphNodeType*) { return cudaErrorNotSupported; }
cudaError_t cudaGraphKernelNodeGetParams(cudaGraphNode_t, cudaKernelNodeParams*) { return cudaErrorNotSupported; }
cudaError_t cudaGraphKernelNodeSetAttribute(cudaGraphNode_t, cudaLaunchAttributeID, const cudaLaunchAttributeValue*) { return cudaErrorNotSupported; }
cudaError_t cudaGraphInstantiateWithFlags(cudaGraphExec_t*, cudaGraph_t, unsigned long long) { return cudaErrorNotSupported; }
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t) { return cudaErrorNotSupported; }
cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }

}  // extern "C"
