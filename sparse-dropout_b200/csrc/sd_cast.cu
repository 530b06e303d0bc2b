// fp32 -> 16-bit copies of a layer's operands under autocast, both operands from one launch.
//
// The reference leaves these casts to torch.autocast (flash_dropout/functional/blockwise_dropout_matmul_cuda.py:9), one
// kernel per tensor and, in backward, one more per gradient; the gradients of the kernels here leave their epilogues in
// fp32 instead, so these copies are all that is left of the casts.
//
// HBM-bound: 6 bytes per element.  Eight elements per thread and step (two 16-byte loads, one 16-byte store), a grid of
// at most eight CTAs per SM striding over both tensors.
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include "sd_common.h"

namespace sd {

constexpr int kCastThreads = 256;

struct CastSeg {
    const float* src;
    void* dst;
    long long n;
};

template <bool BF16>
__device__ __forceinline__ uint32_t cast_pack(float a, float b) {
    if (BF16) {
        __nv_bfloat162 v = __floats2bfloat162_rn(a, b);
        return *reinterpret_cast<uint32_t*>(&v);
    }
    __half2 v = __floats2half2_rn(a, b);
    return *reinterpret_cast<uint32_t*>(&v);
}

template <bool BF16>
__device__ __forceinline__ void cast_seg(const CastSeg& s, long long first, long long stride) {
    const long long n8 = s.n >> 3;
    for (long long i = first; i < n8; i += stride) {
        const float4 a = __ldcs(reinterpret_cast<const float4*>(s.src) + 2 * i);
        const float4 b = __ldcs(reinterpret_cast<const float4*>(s.src) + 2 * i + 1);
        reinterpret_cast<uint4*>(s.dst)[i] = make_uint4(cast_pack<BF16>(a.x, a.y), cast_pack<BF16>(a.z, a.w),
                                                        cast_pack<BF16>(b.x, b.y), cast_pack<BF16>(b.z, b.w));
    }
    if (first < (s.n & 7)) {                                  // the last elements of a length that is no multiple of 8
        const long long i = (n8 << 3) + first;
        const uint32_t v = cast_pack<BF16>(s.src[i], 0.f);
        static_cast<unsigned short*>(s.dst)[i] = (unsigned short)(v & 0xffffu);
    }
}

template <bool BF16>
__global__ void __launch_bounds__(kCastThreads) cast16_kernel(CastSeg a, CastSeg b) {
    const long long first = (long long)blockIdx.x * kCastThreads + threadIdx.x;
    const long long stride = (long long)gridDim.x * kCastThreads;
    cast_seg<BF16>(a, first, stride);
    cast_seg<BF16>(b, first, stride);
}

// y = x + r with x in fp32 and r in 16 bits: a transformer's residual sum under autocast (eval/llm/model.py:80-83).  HBM-bound,
// 10 bytes an element.  torch's kernel for mixed types moves them one element at a time: 21.6 us for 16384 x 384 in bf16, 9.6 here.
template <bool BF16>
__device__ __forceinline__ float2 residual_pair(uint32_t w) {
    if (BF16) return make_float2(__uint_as_float(w << 16), __uint_as_float(w & 0xffff0000u));
    return __half22float2(*reinterpret_cast<const __half2*>(&w));
}
template <bool BF16>
__global__ void __launch_bounds__(kCastThreads) residual_add_kernel(const float* __restrict__ x, const unsigned short* __restrict__ r,
                                                                    float* __restrict__ y, long long n) {
    const long long i = ((long long)blockIdx.x * kCastThreads + threadIdx.x) * 8;
    if (i + 8 <= n) {
        const float4 a = __ldg(reinterpret_cast<const float4*>(x + i)), b = __ldg(reinterpret_cast<const float4*>(x + i) + 1);
        const uint4 w = __ldg(reinterpret_cast<const uint4*>(r + i));
        const float2 p = residual_pair<BF16>(w.x), q = residual_pair<BF16>(w.y), s = residual_pair<BF16>(w.z), t = residual_pair<BF16>(w.w);
        reinterpret_cast<float4*>(y + i)[0] = make_float4(a.x + p.x, a.y + p.y, a.z + q.x, a.w + q.y);
        reinterpret_cast<float4*>(y + i)[1] = make_float4(b.x + s.x, b.y + s.y, b.z + t.x, b.w + t.y);
    } else {
        for (long long k = i; k < n; ++k) y[k] = x[k] + residual_pair<BF16>(r[k]).x;
    }
}

}  // namespace sd

extern "C" int sd_residual_add(const float* x, const void* r, float* y, int64_t n, int dtype, void* stream) {
    if (n < 0 || (n && (!x || !r || !y))) return sd::fail(SD_ERR_INVALID_ARG, "sd_residual_add: null pointer or negative length");
    if (dtype != SD_F16 && dtype != SD_BF16) return sd::fail(SD_ERR_INVALID_ARG, "dtype must be SD_F16 or SD_BF16");
    if ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(r) | reinterpret_cast<uintptr_t>(y)) & 15)
        return sd::fail(SD_ERR_LAYOUT, "sd_residual_add: pointers must be 16-byte aligned");
    if (n == 0) return SD_OK;
    const long long blocks = (n + sd::kCastThreads * 8 - 1) / (sd::kCastThreads * 8);
    if (blocks > (1ll << 31) - 1) return sd::fail(SD_ERR_TOO_LARGE, "sd_residual_add: too many elements");
    auto kernel = dtype == SD_BF16 ? &sd::residual_add_kernel<true> : &sd::residual_add_kernel<false>;
    kernel<<<unsigned(blocks), sd::kCastThreads, 0, static_cast<cudaStream_t>(stream)>>>(x, static_cast<const unsigned short*>(r), y, n);
    SD_CUDA_TRY(cudaGetLastError());
    return SD_OK;
}

extern "C" int sd_cast16(const float* a, void* a16, int64_t na, const float* b, void* b16, int64_t nb, int dtype,
                         void* stream) {
    if (na < 0 || nb < 0 || (na && (!a || !a16)) || (nb && (!b || !b16)))
        return sd::fail(SD_ERR_INVALID_ARG, "sd_cast16: null pointer or negative length");
    if (dtype != SD_F16 && dtype != SD_BF16) return sd::fail(SD_ERR_INVALID_ARG, "dtype must be SD_F16 or SD_BF16");
    if ((reinterpret_cast<uintptr_t>(a) | reinterpret_cast<uintptr_t>(a16) | reinterpret_cast<uintptr_t>(b) |
         reinterpret_cast<uintptr_t>(b16)) & 15)
        return sd::fail(SD_ERR_LAYOUT, "sd_cast16: pointers must be 16-byte aligned");
    const int64_t most = na > nb ? na : nb;
    if (most == 0) return SD_OK;
    int sms = 0;
    if (int rc = sd::sm_count_current_device(&sms)) return rc;
    int64_t grid = (most / 8 + sd::kCastThreads - 1) / sd::kCastThreads;
    if (grid < 1) grid = 1;
    if (grid > int64_t(sms) * 8) grid = int64_t(sms) * 8;
    const sd::CastSeg sa{a, a16, na}, sb{b, b16, nb};
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    if (dtype == SD_BF16) sd::cast16_kernel<true><<<int(grid), sd::kCastThreads, 0, st>>>(sa, sb);
    else sd::cast16_kernel<false><<<int(grid), sd::kCastThreads, 0, st>>>(sa, sb);
    SD_CUDA_TRY(cudaGetLastError());
    return SD_OK;
}
