// GELU, x * Phi(x), forward and backward on 16-bit tensors: the activation between the two SparseDrop layers of a
// transformer MLP (eval/llm/model.py:60-69, eval/vit/model.py:60-66).
//
// torch's own formulas, CDF = (1 + erf(x / sqrt 2)) / 2 and density exp(-x^2 / 2) / sqrt(2 pi), in fp32 with CUDA's erff and
// expf, rounded once: over all finite 16-bit inputs no result is further from fp64 than torch's.  The instructions of
// erff and expf bound both kernels, not the 100 and 151 MB that they move at 16384 x 1536 in bf16 (16 and 23 us of HBM time):
// 29.2-29.8 and 38.4-38.6 us, torch's kernels 29.2 and 40.3.  What was measured against that, same size:
//   Abramowitz & Stegun 7.1.26 with __expf and __fdividef, one exponential for both: 24.2 and 28.3, but twice the error of the
//   derivative (3.2e-7 against 1.3e-7 in fp32), and of the fp16 inputs below 3 eleven values and 18 derivatives rounded
//   further off (one and none nearer);
//   CDF = erfc(-x / sqrt 2) / 2, which keeps the far negative tail's leading digits: 44.8 and 52.6.
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include "sd_common.h"

namespace sd {

constexpr int kGeluThreads = 256, kGeluVec = 8;               // eight elements, 16 bytes of each tensor, per thread

template <bool IS_BF16>
__device__ __forceinline__ float2 widen(uint32_t w) {
    if (IS_BF16) return make_float2(__uint_as_float(w << 16), __uint_as_float(w & 0xffff0000u));
    return __half22float2(*reinterpret_cast<const __half2*>(&w));
}
template <bool IS_BF16>
__device__ __forceinline__ uint32_t narrow(float a, float b) {
    if (IS_BF16) {
        const __nv_bfloat162 v = __floats2bfloat162_rn(a, b);
        return *reinterpret_cast<const uint32_t*>(&v);
    }
    const __half2 v = __floats2half2_rn(a, b);
    return *reinterpret_cast<const uint32_t*>(&v);
}

template <bool BACKWARD>
__device__ __forceinline__ float gelu_one(float x, float dy) {
    const float cdf = 0.5f * (1.f + erff(x * 0.70710678118654752f));
    if (!BACKWARD) return x * cdf;                            // infinities and NaN come out as from torch
    return dy * (cdf + x * (expf(-0.5f * x * x) * 0.39894228040143268f));
}

template <bool IS_BF16, bool BACKWARD>
__global__ void __launch_bounds__(kGeluThreads) gelu_kernel(const unsigned short* __restrict__ x, const unsigned short* __restrict__ dy,
                                                            unsigned short* __restrict__ out, long long n) {
    const long long i = ((long long)blockIdx.x * kGeluThreads + threadIdx.x) * kGeluVec;
    if (i + kGeluVec <= n) {
        const uint4 xv = __ldg(reinterpret_cast<const uint4*>(x + i));
        uint4 dv = make_uint4(0, 0, 0, 0), o;
        if (BACKWARD) dv = __ldg(reinterpret_cast<const uint4*>(dy + i));
        const uint32_t xs[4] = {xv.x, xv.y, xv.z, xv.w}, ds[4] = {dv.x, dv.y, dv.z, dv.w};
        uint32_t r[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const float2 a = widen<IS_BF16>(xs[j]), d = widen<IS_BF16>(ds[j]);
            r[j] = narrow<IS_BF16>(gelu_one<BACKWARD>(a.x, d.x), gelu_one<BACKWARD>(a.y, d.y));
        }
        o = make_uint4(r[0], r[1], r[2], r[3]);
        *reinterpret_cast<uint4*>(out + i) = o;
    } else {
        for (long long k = i; k < n; ++k) {
            const float d = BACKWARD ? widen<IS_BF16>(dy[k]).x : 0.f;
            out[k] = (unsigned short)narrow<IS_BF16>(gelu_one<BACKWARD>(widen<IS_BF16>(x[k]).x, d), 0.f);
        }
    }
}

static int run_gelu(const void* x, const void* dy, void* out, int64_t n, int dtype, cudaStream_t st) {
    if (n == 0) return SD_OK;
    if (n < 0 || !x || !out) return fail(SD_ERR_INVALID_ARG, "sd_gelu: bad arguments");
    if (dtype != SD_F16 && dtype != SD_BF16) return fail(SD_ERR_INVALID_ARG, "dtype must be SD_F16 or SD_BF16");
    if ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(dy) | reinterpret_cast<uintptr_t>(out)) & 15)
        return fail(SD_ERR_LAYOUT, "sd_gelu: tensors must be 16-byte aligned");
    const long long blocks = (n + kGeluThreads * kGeluVec - 1) / (kGeluThreads * kGeluVec);
    if (blocks > (1ll << 31) - 1) return fail(SD_ERR_TOO_LARGE, "sd_gelu: too many elements");
    auto kernel = dtype == SD_BF16 ? (dy ? &gelu_kernel<true, true> : &gelu_kernel<true, false>)
                                   : (dy ? &gelu_kernel<false, true> : &gelu_kernel<false, false>);
    kernel<<<unsigned(blocks), kGeluThreads, 0, st>>>(static_cast<const unsigned short*>(x), static_cast<const unsigned short*>(dy),
                                                      static_cast<unsigned short*>(out), n);
    SD_CUDA_TRY(cudaGetLastError());
    return SD_OK;
}

}  // namespace sd

extern "C" {

int sd_gelu_fwd(const void* x, void* y, int64_t n, int dtype, void* stream) {
    return sd::run_gelu(x, nullptr, y, n, dtype, static_cast<cudaStream_t>(stream));
}

int sd_gelu_bwd(const void* dy, const void* x, void* dx, int64_t n, int dtype, void* stream) {
    if (!dy && n) return sd::fail(SD_ERR_INVALID_ARG, "sd_gelu_bwd: dy is null");
    return sd::run_gelu(x, dy, dx, n, dtype, static_cast<cudaStream_t>(stream));
}

}  // extern "C"
