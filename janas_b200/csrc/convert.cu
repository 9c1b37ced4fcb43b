// Element type conversions on the device: bfloat16 <-> float32 (0: float32,
// 1: bfloat16, as everywhere in the kernels' C interface).  Used when weights of
// different stored types are fused into one matrix.  And the copy of a step's few
// words between pinned host memory and the device.
#include "common.cuh"
#include "kernels.h"

namespace {

template <typename S, typename D>
__global__ void convert_kernel(const S *__restrict__ src, D *__restrict__ dst, long long n)
{
    long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    long long step = (long long)gridDim.x * blockDim.x;
    for (; i < n; i += step) {
        float v;
        if constexpr (sizeof(S) == 4)
            v = src[i];
        else
            v = __bfloat162float(src[i]);
        if constexpr (sizeof(D) == 4)
            dst[i] = v;
        else
            dst[i] = __float2bfloat16_rn(v);
    }
}

// dst[i] = src[i], a word a thread, either side pinned host memory.  The words of the host are on their way before the
// kernel ahead has ended (src_early: nothing on the stream writes src).  Never allows the kernel behind it to start early,
// and no thread ends before its word can be read by the whole device: kernels read a step's positions and tables ahead of
// their own waits (see common.cuh: pdl_wait), and only the kernel right behind this one could wait for its end.
__global__ void __launch_bounds__(256)
copy_words_kernel(const uint32_t *src, uint32_t *dst, int n, int src_early)
{
    int i = blockIdx.x * 256 + threadIdx.x;
    uint32_t v = 0;
    if (src_early && i < n)
        v = __ldcv(src + i);
    jb::pdl_wait();
    if (!src_early && i < n)
        v = __ldcv(src + i);
    if (i < n)
        __stcg(dst + i, v);
    __threadfence();
}

}  // namespace

// n words from or to pinned host memory by a kernel: a copy between two kernels of a stream goes through a copy engine,
// which costs 5 to 9 us of hand-overs each way.  Two of them a decode step: 17 steps of 8 sequences over four layers 5,248 -> 5,115
// us, nine of 64 sequences 4,997 -> 4,909.
extern "C" int jb_copy_words(const void *src, void *dst, int n, int src_early, cudaStream_t st)
{
    if (n <= 0)
        return jb::JB_OK;
    if ((uintptr_t)src % 4 || (uintptr_t)dst % 4)
        return jb::JB_EINVAL;
    jb::launch(copy_words_kernel, (unsigned)((n + 255) / 256), 256, 0, st, (const uint32_t *)src, (uint32_t *)dst, n, src_early);
    return jb::launch_status();
}

extern "C" int jb_convert(const void *src, int src_dt, void *dst, int dst_dt, long long n,
                          cudaStream_t st)
{
    if (n <= 0)
        return 0;
    if ((src_dt != 0 && src_dt != 1) || (dst_dt != 0 && dst_dt != 1))
        return -1;
    long long b = (n + 255) / 256;
    unsigned blocks = (unsigned)(b > 148 * 16 ? 148 * 16 : b);
    if (src_dt == dst_dt) {
        size_t bytes = (size_t)n * (src_dt == 0 ? 4 : 2);
        return cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDeviceToDevice, st) == cudaSuccess ? 0 : -2;
    }
    if (src_dt == 1)
        convert_kernel<<<blocks, 256, 0, st>>>((const __nv_bfloat16 *)src, (float *)dst, n);
    else
        convert_kernel<<<blocks, 256, 0, st>>>((const float *)src, (__nv_bfloat16 *)dst, n);
    return cudaGetLastError() == cudaSuccess ? 0 : -2;
}
