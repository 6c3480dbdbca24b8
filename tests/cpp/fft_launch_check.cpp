/* The launches of the FP64 transforms (csrc/sh_fft*.cu) against a stand-in
 * for the CUDA runtime that keeps, as the runtime does, the dynamic
 * shared-memory limit of a kernel per device.  For every grid size: the first
 * transform of a process on device 0, then one on device 1, then one whose
 * limit cannot be set and the same again; and the stream on which the twiddle
 * factors are copied.  Linked with the library's objects; no GPU. */
#include <cuda_runtime.h>

#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <map>
#include <utility>

#include "sh_fft.h"

namespace {
int device = 0;
bool refuse = false; /* setting a limit fails */
std::map<std::pair<int, const void *>, int> limit;
cudaError_t last = cudaSuccess;
long long launched = 0;
cudaStream_t copied_on = nullptr;
struct {
    dim3 grid, block;
    size_t smem;
    void *stream;
} config;
} // namespace

extern "C" {
void **__cudaRegisterFatBinary(void *) {
    static void *handle;
    return &handle;
}
void __cudaRegisterFatBinaryEnd(void **) {}
void __cudaUnregisterFatBinary(void **) {}
void __cudaRegisterFunction(void **, const char *, char *, const char *, int, uint3 *, uint3 *,
                            dim3 *, dim3 *, int *) {}
unsigned __cudaPushCallConfiguration(dim3 grid, dim3 block, size_t smem, void *stream) {
    config = {grid, block, smem, stream};
    return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3 *grid, dim3 *block, size_t *smem, void *stream) {
    *grid = config.grid;
    *block = config.block;
    *smem = config.smem;
    *(void **)stream = config.stream;
    return cudaSuccess;
}
cudaError_t __cudaGetKernel(cudaKernel_t *kernel, const void *fn) {
    *kernel = (cudaKernel_t)fn;
    return cudaSuccess;
}
cudaError_t __cudaLaunchKernel(cudaKernel_t kernel, dim3, dim3, void **, size_t smem,
                               cudaStream_t) {
    /* 48 KB without the attribute, with what the kernel has of its own */
    const auto it = limit.find({device, (const void *)kernel});
    const size_t most = it == limit.end() ? 48 * 1024 - 17 * 25 * 8 : (size_t)it->second;
    if (smem > most) return last = cudaErrorInvalidValue;
    ++launched;
    return cudaSuccess;
}
cudaError_t cudaFuncSetAttribute(const void *fn, cudaFuncAttribute attr, int value) {
    if (refuse) return last = cudaErrorInvalidValue;
    if (attr == cudaFuncAttributeMaxDynamicSharedMemorySize) limit[{device, fn}] = value;
    return cudaSuccess;
}
cudaError_t cudaGetLastError() {
    const cudaError_t e = last;
    last = cudaSuccess;
    return e;
}
cudaError_t cudaMalloc(void **p, size_t n) {
    *p = std::malloc(n);
    return cudaSuccess;
}
cudaError_t cudaFree(void *p) {
    std::free(p);
    return cudaSuccess;
}
/* a copy on the default stream: other streams' kernels do not wait for it */
cudaError_t cudaMemcpy(void *, const void *, size_t, cudaMemcpyKind) {
    copied_on = nullptr;
    return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void *d, const void *h, size_t n, cudaMemcpyKind, cudaStream_t s) {
    std::memcpy(d, h, n);
    copied_on = s;
    return cudaSuccess;
}
}

int main() {
    int bad = 0;
    auto check = [&](int P, const char *what, bool want) {
        const long long before = launched;
        const cudaError_t e = sh::fft::transform3(nullptr, 3, P, nullptr, nullptr);
        const bool ok = want ? e == cudaSuccess && launched == before + 3 : e != cudaSuccess;
        if (!ok) {
            std::printf("P = %d, %s: error %d, %lld launches\n", P, what, (int)e,
                        launched - before);
            ++bad;
        }
        last = cudaSuccess;
    };
    int sizes = 0;
    for (int P = 1; P <= 512; ++P) {
        if (!sh::fft::supported(P)) continue;
        ++sizes;
        device = 0;
        check(P, "device 0", true);
        device = 1;
        check(P, "device 1 of the same process", true);
        if (P >= 192) { /* more than 48 KB */
            device = 2;
            refuse = true;
            check(P, "a limit that cannot be set", false);
            refuse = false;
            check(P, "the call after it", true);
        }
    }
    /* the twiddle factors, in the order of the stream that reads them */
    const cudaStream_t stream = (cudaStream_t)&sizes;
    sh::fft::Twiddle *const t = sh::fft::make_table(64, stream);
    const sh::fft::Twiddle want = sh::fft::make_twiddle(5, 64);
    if (!t || copied_on != stream || std::memcmp(&t[5], &want, sizeof want) != 0) {
        std::printf("twiddle factors not written on the stream\n");
        ++bad;
    }
    cudaFree(t);
    std::printf("%d sizes\n", sizes);
    return bad || sizes == 0;
}
