// The library's scratch pool (scratch.cuh).

#include "scratch.cuh"

#include <mutex>

namespace sxb {
namespace {

constexpr uint64_t kKeepBytes = 1ull << 30;  // a 4096-token prefill of 4096-wide activations in ten slots is 335 MB
constexpr int kMaxDevices = 64;

std::mutex g_mutex;
cudaMemPool_t g_pool[kMaxDevices] = {};
thread_local int g_refuse = 0;

// The current device's pool, created on first use.
cudaMemPool_t pool() {
    int dev = -1;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return nullptr;
    std::lock_guard<std::mutex> lock(g_mutex);
    if (g_pool[dev] == nullptr) {
        cudaMemPoolProps props = {};
        props.allocType = cudaMemAllocationTypePinned;
        props.location.type = cudaMemLocationTypeDevice;
        props.location.id = dev;
        cudaMemPool_t p = nullptr;
        if (cudaMemPoolCreate(&p, &props) != cudaSuccess) return nullptr;
        uint64_t keep = kKeepBytes;
        if (cudaMemPoolSetAttribute(p, cudaMemPoolAttrReleaseThreshold, &keep) != cudaSuccess) {
            cudaMemPoolDestroy(p);
            return nullptr;
        }
        g_pool[dev] = p;
    }
    return g_pool[dev];
}

}  // namespace

bool StreamScratch::get(size_t bytes, cudaStream_t stream) {
    if (g_refuse > 0 || p_ != nullptr) return false;
    // An error that the caller's earlier calls left pending is for the next launch check to report: nothing here may replace or
    // clear it.  Past this line a pending error is this function's own.
    if (cudaPeekAtLastError() != cudaSuccess) return false;
    // Not under capture: the allocation would be a node of the graph, which then can no longer be cloned, be a child of another or
    // have two executable instances, and whose memory is neither bounded by this pool nor given back by sxb_release_scratch.
    cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(stream, &capture) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    if (capture != cudaStreamCaptureStatusNone) return false;
    cudaMemPool_t from = pool();
    if (from == nullptr || cudaMallocFromPoolAsync(&p_, bytes, from, stream) != cudaSuccess) {
        p_ = nullptr;
        cudaGetLastError();  // the caller has another way
        return false;
    }
    stream_ = stream;
    return true;
}

StreamScratch::~StreamScratch() {
    if (p_ != nullptr) cudaFreeAsync(p_, stream_);
}

NoScratch::NoScratch() { ++g_refuse; }
NoScratch::~NoScratch() { --g_refuse; }

}  // namespace sxb

extern "C" int sxb_release_scratch(void) {
    using namespace sxb;
    int dev = -1;
    SXB_CUDA(cudaGetDevice(&dev), "release_scratch: no current device");
    std::lock_guard<std::mutex> lock(g_mutex);
    if (dev >= 0 && dev < kMaxDevices && g_pool[dev] != nullptr) SXB_CUDA(cudaMemPoolTrimTo(g_pool[dev], 0), "release_scratch");
    return SXB_OK;
}
