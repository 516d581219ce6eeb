// Library-level entry points: version, error strings, shared host helpers.
#include <math.h>
#include <stdio.h>
#include <string.h>

#include <algorithm>
#include <atomic>
#include <map>
#include <mutex>
#include <utility>

#include "hgb_common.cuh"

namespace {

__global__ void k_sqrt(double *x, long n) {
    long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) x[i] = sqrt(x[i]);
}

// Host words in a kernel's arguments, which the launch (or the capture of it) copies: their source may go
// when the call returns.  cudaMemcpyAsync promises that of pageable memory only where it stages the copy, and
// a device that addresses host memory need not.
template <int WORDS>
struct HostWords {
    uint32_t w[WORDS];
};
template <int WORDS>
__global__ void k_put_words(const __grid_constant__ HostWords<WORDS> h, uint32_t *dst, int n) {
    const int i = (int)(blockIdx.x * blockDim.x + threadIdx.x);
    if (i < n) dst[i] = h.w[i];
}

template <int WORDS>
void put_words(uint32_t *dst, const char *host, int n, cudaStream_t st) {
    HostWords<WORDS> h;
    memcpy(h.w, host, sizeof(uint32_t) * n);
    k_put_words<WORDS><<<(unsigned)hgb::ceil_div(n, 128), 128, 0, st>>>(h, dst, n);
}

}  // namespace

namespace hgb {

int upload_words(void *dst, const void *host, size_t bytes, cudaStream_t st) {
    constexpr int MOST = 8000;   // words of one launch: its arguments stay below 32,764 bytes
    for (size_t at = 0; at < bytes; at += sizeof(uint32_t) * MOST) {
        const int n = (int)(std::min(bytes - at, sizeof(uint32_t) * MOST) / sizeof(uint32_t));
        uint32_t *d = (uint32_t *)((char *)dst + at);
        const char *h = (const char *)host + at;
        // (arguments are copied whole: 32,000 bytes of them cost the host 2 us more than 4,000)
        if (n <= 250) put_words<250>(d, h, n, st);
        else if (n <= 1000) put_words<1000>(d, h, n, st);
        else put_words<MOST>(d, h, n, st);
        const int rc = check_launch();
        if (rc) return rc;
    }
    return HGB_OK;
}

static thread_local char g_last_cuda_error[256] = "";

void set_cuda_error(cudaError_t err) {
    snprintf(g_last_cuda_error, sizeof(g_last_cuda_error), "%s: %s", cudaGetErrorName(err),
             cudaGetErrorString(err));
}

int check_launch() {
    cudaError_t err = cudaGetLastError();
    if (err != cudaSuccess) {
        set_cuda_error(err);
        return HGB_ERR_CUDA;
    }
    return HGB_OK;
}

int sm_count() {
    static std::atomic<int> cache[64];
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 152;
    int n = cache[dev].load(std::memory_order_relaxed);
    if (n > 0) return n;
    if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0) n = 152;
    cache[dev].store(n, std::memory_order_relaxed);
    return n;
}

int ensure_dyn_smem(const void *func, size_t bytes) {
    static std::mutex mu;
    static std::map<std::pair<const void *, int>, size_t> raised;   // (function, device) -> cap set
    if (bytes == 0) return HGB_OK;
    int dev = 0;
    cudaError_t err = cudaGetDevice(&dev);
    if (err != cudaSuccess) {
        set_cuda_error(err);
        return HGB_ERR_CUDA;
    }
    std::lock_guard<std::mutex> lock(mu);
    size_t &cap = raised[std::make_pair(func, dev)];
    if (cap == 0) {
        // once, to all that the device gives the function (its default, 48 KB, counts its static shared
        // memory too)
        cudaFuncAttributes fa;
        int most = 0;
        err = cudaDeviceGetAttribute(&most, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
        if (err == cudaSuccess) err = cudaFuncGetAttributes(&fa, func);
        if (err == cudaSuccess) {
            most -= (int)fa.sharedSizeBytes;
            err = cudaFuncSetAttribute(func, cudaFuncAttributeMaxDynamicSharedMemorySize, most);
        }
        if (err != cudaSuccess) {
            set_cuda_error(err);
            return HGB_ERR_CUDA;
        }
        cap = (size_t)most;
    }
    if (bytes <= cap) return HGB_OK;
    set_cuda_error(cudaErrorInvalidValue);   // as raising the cap beyond the device's limit
    return HGB_ERR_CUDA;
}

CyConst cy_const() {
    CyConst c;
    c.c_dadt = -64.0 * pow(HGB_CY_NWTG, 3) / 5.0 / pow(HGB_CY_SPLC, 5);
    c.kfreq = (1.0 / (2.0 * M_PI)) * sqrt(HGB_CY_NWTG);
    c.ksepa = pow(HGB_CY_NWTG, 1.0 / 3.0) / pow(2.0 * M_PI, 2.0 / 3.0);
    c.fourpi = 4 * M_PI * HGB_CY_SPLC / HGB_CY_MPC;
    return c;
}

}  // namespace hgb

extern "C" {

int hgb_version(void) { return 1; }

const char *hgb_error_string(int code) {
    switch (code) {
        case HGB_OK: return "success";
        case HGB_ERR_INVALID_ARGUMENT: return "invalid argument";
        case HGB_ERR_CUDA: return "CUDA error";
        case HGB_ERR_WORKSPACE: return "workspace too small";
        case HGB_ERR_CAPACITY: return "input exceeds the static scratch capacity";
        case HGB_ERR_DEVICE_LIMIT: return "a bounded device wait gave up; outputs not valid";
        default: return "unknown error";
    }
}

const char *hgb_last_cuda_error(void) { return hgb::g_last_cuda_error; }

int hgb_upload(void *dst, const void *host, size_t bytes, void *stream) {
    if ((bytes && (!dst || !host)) || (bytes & 3) || ((uintptr_t)dst & 3)) return HGB_ERR_INVALID_ARGUMENT;
    return hgb::upload_words(dst, host, bytes, (cudaStream_t)stream);
}

int hgb_sqrt_inplace(double *x, long n, void *stream) {
    if (!x || n < 0) return HGB_ERR_INVALID_ARGUMENT;
    if (n == 0) return HGB_OK;
    k_sqrt<<<(unsigned)hgb::ceil_div(n, 256), 256, 0, (cudaStream_t)stream>>>(x, n);
    return hgb::check_launch();
}

}  // extern "C"
