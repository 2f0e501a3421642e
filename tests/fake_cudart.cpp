// A stand-in for the CUDA runtime, preloaded over libcudart so that the
// library's host code runs without a GPU.  Device memory is host memory and
// kernels do nothing, but for the few whose outputs steer the host.  A copy to
// the device may read its source until the stream is synchronised, as the
// runtime allows it to: at each synchronisation the sources of the copies before
// it are compared with what they held at the call.
#include <cuda_runtime_api.h>
#include <sys/uio.h>
#include <unistd.h>

#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <map>
#include <mutex>
#include <string>
#include <vector>

#undef cudaGetDeviceProperties

namespace {
struct Copy {
    cudaStream_t stream;
    const void* src;
    std::vector<char> held;
};
std::mutex mu;
std::vector<Copy>& copies() { static std::vector<Copy> v; return v; }
std::map<const void*, std::string>& names() { static std::map<const void*, std::string> m; return m; }
std::map<std::string, long>& launches() { static std::map<std::string, long> m; return m; }
std::map<char*, size_t>& pinned() { static std::map<char*, size_t> m; return m; }
long changed = 0, read_back = 0, allocations = 0, fail_in = 0;
thread_local cudaError_t last_error = cudaSuccess;
struct Call { dim3 grid, block; size_t smem; void* stream; };
thread_local std::vector<Call> calls;

void finish(bool all, cudaStream_t s) {
    std::lock_guard<std::mutex> lock(mu);
    std::vector<Copy> rest;
    for (Copy& c : copies()) {
        if (!all && c.stream != s) {
            rest.push_back(std::move(c));
            continue;
        }
        std::vector<char> now(c.held.size());
        iovec to{now.data(), now.size()}, from{const_cast<void*>(c.src), now.size()};
        const ssize_t n = process_vm_readv(getpid(), &to, 1, &from, 1, 0);  // fails where nothing is mapped
        ++read_back;
        if (n != (ssize_t)now.size() || std::memcmp(now.data(), c.held.data(), now.size()) != 0) ++changed;
    }
    copies().swap(rest);
}

void launch(const void* fn, void** args) {
    std::string name;
    {
        std::lock_guard<std::mutex> lock(mu);
        name = names()[fn];
        ++launches()[name];
    }
    if (name.find("k_jacobi_svd") != std::string::npos) {  // the identity, descending eigenvalues
        const int a = *(int*)args[1];
        double *V = *(double**)args[2], *sig = *(double**)args[3];
        for (int i = 0; i < a; ++i) {
            sig[i] = a - i;
            for (int j = 0; j < a; ++j) V[i * a + j] = i == j;
        }
    } else if (name.find("6k_drawE") != std::string::npos) {  // tail draws for the host
        struct Tails { unsigned long long drawn; unsigned n, undecided; struct { uint64_t slot; double a; } e[1]; };
        const unsigned cap = *(unsigned*)args[2];
        Tails* t = *(Tails**)args[5];
        t->drawn = 1ull << 62;
        t->n = cap;
        for (unsigned i = 0; i < cap; ++i) {
            t->e[i].slot = 2 * i;
            t->e[i].a = 0.5;
        }
    }
}
}  // namespace

extern "C" {
// for the test
long fake_changed_sources() { return changed; }
long fake_sources_compared() { return read_back; }
long fake_pending() { return (long)copies().size(); }
// the n-th allocation of device memory from here on fails (0: none)
void fake_fail_allocation(long n) { allocations = 0, fail_in = n; }
long fake_allocations() { return allocations; }
long fake_launches(const char* part) {
    std::lock_guard<std::mutex> lock(mu);
    long n = 0;
    for (const auto& l : launches())
        if (l.first.find(part) != std::string::npos) n += l.second;
    return n;
}

void** __cudaRegisterFatBinary(void*) { static void* h; return &h; }
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterVar(void**, char*, char*, const char*, int, size_t, int, int) {}
void __cudaRegisterFunction(void**, const char* host, char*, const char* name, int, void*, void*, void*, void*, int*) {
    names()[host] = name;
}
unsigned __cudaPushCallConfiguration(dim3 g, dim3 b, size_t smem, void* s) {
    calls.push_back({g, b, smem, s});
    return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3* g, dim3* b, size_t* smem, void* s) {
    *g = calls.back().grid, *b = calls.back().block, *smem = calls.back().smem, *(void**)s = calls.back().stream;
    calls.pop_back();
    return cudaSuccess;
}
cudaError_t __cudaGetKernel(cudaKernel_t* k, const void* fn) {
    *k = (cudaKernel_t)fn;
    return cudaSuccess;
}
cudaError_t __cudaLaunchKernel(cudaKernel_t k, dim3, dim3, void** args, size_t, cudaStream_t) {
    launch((const void*)k, args);
    return cudaSuccess;
}
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t*, const void* fn, void** args) {
    launch(fn, args);
    return cudaSuccess;
}

cudaError_t cudaGetDeviceCount(int* n) { *n = 1; return cudaSuccess; }
cudaError_t cudaGetDevice(int* d) { *d = 0; return cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr, int) { *v = 0; return cudaSuccess; }
cudaError_t cudaGetDeviceProperties(cudaDeviceProp* p, int) {
    std::memset(p, 0, sizeof *p);
    p->major = 10, p->minor = 3, p->multiProcessorCount = 152;
    return cudaSuccess;
}
cudaError_t cudaDeviceGetDefaultMemPool(cudaMemPool_t* p, int) { *p = nullptr; return cudaSuccess; }
cudaError_t cudaMemPoolSetAttribute(cudaMemPool_t, cudaMemPoolAttr, void*) { return cudaSuccess; }
cudaError_t cudaFuncGetAttributes(cudaFuncAttributes* a, const void*) { std::memset(a, 0, sizeof *a); return cudaSuccess; }
cudaError_t cudaFuncSetAttribute(const void*, cudaFuncAttribute, int) { return cudaSuccess; }
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int* n, const void*, int, size_t, unsigned) {
    *n = 1;
    return cudaSuccess;
}
cudaError_t cudaGetSymbolAddress(void** p, const void*) {
    static char hist[16 << 20];
    *p = hist;
    return cudaSuccess;
}
cudaError_t cudaGetDriverEntryPointByVersion(const char*, void** f, unsigned, unsigned long long,
                                             cudaDriverEntryPointQueryResult* r) {
    *f = nullptr;
    if (r) *r = cudaDriverEntryPointSymbolNotFound;
    return cudaErrorNotSupported;
}
const char* cudaGetErrorString(cudaError_t) { return "error of the stand-in runtime"; }
cudaError_t cudaGetLastError() {
    const cudaError_t e = last_error;
    last_error = cudaSuccess;
    return e;
}
cudaError_t cudaPeekAtLastError() { return last_error; }

cudaError_t cudaMallocAsync(void** p, size_t n, cudaStream_t) {
    {
        std::lock_guard<std::mutex> lock(mu);
        if (++allocations == fail_in) return last_error = cudaErrorMemoryAllocation;
    }
    *p = std::calloc(1, n + 4096);
    return *p ? cudaSuccess : cudaErrorMemoryAllocation;
}
cudaError_t cudaFreeAsync(void* p, cudaStream_t) { std::free(p); return cudaSuccess; }
cudaError_t cudaMallocHost(void** p, size_t n) {
    *p = std::calloc(1, n);
    std::lock_guard<std::mutex> lock(mu);
    pinned()[(char*)*p] = n;
    return cudaSuccess;
}
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) { return cudaMallocHost(p, n); }
cudaError_t cudaFreeHost(void* p) {
    std::lock_guard<std::mutex> lock(mu);
    pinned().erase((char*)p);
    std::free(p);
    return cudaSuccess;
}
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes* a, const void* p) {
    std::memset(a, 0, sizeof *a);
    a->type = cudaMemoryTypeUnregistered;
    std::lock_guard<std::mutex> lock(mu);
    for (const auto& r : pinned())
        if ((const char*)p >= r.first && (const char*)p < r.first + r.second) a->type = cudaMemoryTypeHost;
    return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void* dst, const void* src, size_t n, cudaMemcpyKind kind, cudaStream_t s) {
    std::memcpy(dst, src, n);
    if (kind == cudaMemcpyHostToDevice) {
        std::lock_guard<std::mutex> lock(mu);
        copies().push_back({s, src, std::vector<char>((const char*)src, (const char*)src + n)});
    }
    return cudaSuccess;
}
cudaError_t cudaMemcpy2DAsync(void* dst, size_t dp, const void* src, size_t sp, size_t w, size_t h, cudaMemcpyKind,
                              cudaStream_t) {
    for (size_t i = 0; i < h; ++i) std::memcpy((char*)dst + i * dp, (const char*)src + i * sp, w);
    return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void* p, int v, size_t n, cudaStream_t) { std::memset(p, v, n); return cudaSuccess; }

cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) { *s = (cudaStream_t) new int; return cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t s) { finish(false, s); return cudaSuccess; }
cudaError_t cudaDeviceSynchronize() { finish(true, nullptr); return cudaSuccess; }
cudaError_t cudaStreamIsCapturing(cudaStream_t, cudaStreamCaptureStatus* s) {
    *s = cudaStreamCaptureStatusNone;
    return cudaSuccess;
}
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
// an event stands for the stream of its last record
cudaError_t cudaEventCreate(cudaEvent_t* e) { *e = (cudaEvent_t) new cudaStream_t(nullptr); return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { return cudaEventCreate(e); }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s) { *(cudaStream_t*)e = s; return cudaSuccess; }
// (what was enqueued behind the record counts as copied too: the checks are the fewer)
cudaError_t cudaEventSynchronize(cudaEvent_t e) { finish(false, *(cudaStream_t*)e); return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) { *ms = 0.f; return cudaSuccess; }
}
