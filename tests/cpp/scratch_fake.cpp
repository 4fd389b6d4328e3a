// csrc/scratch.cu against a fake runtime, on the CPU: prints one line per check and returns the number of failures.
// Built with the host compiler and no CUDA library; the runtime's entry points that scratch.cu calls are defined here, and the
// two device functions that common.cuh's device helpers mention are declared.
#include <cmath>
unsigned atomicCAS(unsigned *, unsigned, unsigned);
float __int_as_float(int);
#include "../../strixite_b200/csrc/scratch.cu"

#include <cstdio>
#include <thread>

namespace {
cudaError_t g_last = cudaSuccess;           // the runtime's last error
cudaStreamCaptureStatus g_capture = cudaStreamCaptureStatusNone;
bool g_alloc_fails = false, g_query_fails = false;
int g_pools = 0, g_allocs = 0, g_frees = 0, g_trims = 0;
uint64_t g_keep = 0;
cudaStream_t g_freed_on = nullptr;
cudaError_t failed(cudaError_t e) { return g_last = e; }
}  // namespace

extern "C" {
cudaError_t cudaGetLastError() { const cudaError_t e = g_last; g_last = cudaSuccess; return e; }
cudaError_t cudaPeekAtLastError() { return g_last; }
const char *cudaGetErrorString(cudaError_t) { return ""; }
const char *cudaGetErrorName(cudaError_t) { return ""; }
cudaError_t cudaGetDevice(int *d) { *d = 0; return cudaSuccess; }
cudaError_t cudaMemPoolCreate(cudaMemPool_t *p, const cudaMemPoolProps *) { ++g_pools; *p = reinterpret_cast<cudaMemPool_t>(0x10); return cudaSuccess; }
cudaError_t cudaMemPoolDestroy(cudaMemPool_t) { return cudaSuccess; }
cudaError_t cudaMemPoolSetAttribute(cudaMemPool_t, cudaMemPoolAttr, void *v) { g_keep = *static_cast<uint64_t *>(v); return cudaSuccess; }
cudaError_t cudaMemPoolTrimTo(cudaMemPool_t, size_t) { ++g_trims; return cudaSuccess; }
cudaError_t cudaMallocFromPoolAsync(void **p, size_t, cudaMemPool_t, cudaStream_t) {
    if (g_alloc_fails) return failed(cudaErrorMemoryAllocation);
    ++g_allocs;
    *p = reinterpret_cast<void *>(0x1000);
    return cudaSuccess;
}
cudaError_t cudaFreeAsync(void *, cudaStream_t s) { ++g_frees; g_freed_on = s; return cudaSuccess; }
cudaError_t cudaStreamIsCapturing(cudaStream_t, cudaStreamCaptureStatus *s) {
    if (g_query_fails) return failed(cudaErrorStreamCaptureImplicit);
    *s = g_capture;
    return cudaSuccess;
}
}  // extern "C"

namespace sxb {  // errors.cu's, for the C entry
std::string &last_error() { static std::string s; return s; }
int fail_check(const char *, int, const char *, const char *, const std::string &) { return 1; }
int fail_cuda(const char *, int, const char *, cudaError_t, const std::string &) { return 2; }
}  // namespace sxb

int failures = 0;
void check(const char *what, bool ok) {
    std::printf("%s %s\n", ok ? "ok  " : "FAIL", what);
    failures += !ok;
}

int main() {
    const cudaStream_t s = reinterpret_cast<cudaStream_t>(0x20);
    using sxb::StreamScratch;
    g_capture = cudaStreamCaptureStatusActive;
    {
        StreamScratch m;
        check("a captured call gets none, and makes no pool", !m.get(100, s) && m.ptr() == nullptr && g_pools == 0 && g_allocs == 0);
    }
    check("nothing to free after it", g_frees == 0);
    g_capture = cudaStreamCaptureStatusNone, g_query_fails = true;
    {
        StreamScratch m;
        check("none where the capture state cannot be told, and no error left", !m.get(100, s) && g_last == cudaSuccess && g_allocs == 0);
    }
    g_query_fails = false, g_last = cudaErrorInvalidValue;
    {
        StreamScratch m;
        m.get(100, s);
        check("a caller's pending error is still pending", g_last == cudaErrorInvalidValue);
    }
    g_last = cudaErrorInvalidValue, g_alloc_fails = true;
    {
        StreamScratch m;
        check("also where the allocation fails", !m.get(100, s) && g_last == cudaErrorInvalidValue);
    }
    g_last = cudaSuccess;
    {
        StreamScratch m;
        check("an allocation that fails leaves no error behind", !m.get(100, s) && m.ptr() == nullptr && g_last == cudaSuccess);
    }
    g_alloc_fails = false;
    const int frees = g_frees;
    {
        StreamScratch m;
        check("otherwise there is some", m.get(100, s) && m.ptr() != nullptr);
        check("once", !m.get(100, s));
    }
    check("freed on its stream", g_frees == frees + 1 && g_freed_on == s);
    check("one pool, which keeps 1 GiB", g_pools == 1 && g_keep == (1ull << 30));
    {
        const sxb::NoScratch none;
        StreamScratch m;
        check("none inside a NoScratch", !m.get(100, s));
        bool other = false;
        std::thread([&] { StreamScratch t; other = t.get(100, s); }).join();
        check("which is this thread's alone", other);
    }
    StreamScratch after;
    check("some again after it", after.get(100, s));
    check("release trims the pool", sxb_release_scratch() == 0 && g_trims == 1);
    return failures;
}
