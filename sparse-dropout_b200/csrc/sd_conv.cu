// im2col / col2im stages of the SparseDrop convolution, restricted to the kept 128x128 blocks.
//
// The im2col matrix of flash_dropout/functional/im2col_conv2d.py:17-20 has M = N*P*Q rows and K = C*R*S
// columns, k = c*R*S + r*S + s.  It is stored K-outer here ("colT": row k holds all M entries of column k,
// leading dimension ldm), because consecutive m are consecutive pixels of the NCHW input, so both the gather
// and the store run along the contiguous direction and the GEMM kernel takes colT.T as an MN-major operand.
// Only blocks the plan keeps are ever written or read: at p = 0.5 half of the 2 x 302 MB an unfold
// (flash_dropout/functional/im2col_conv2d.py:17) moves.  Both kernels are pure data movement: HBM-bound.
//
// The reference's own CUDA im2col (flash_dropout/cuda/src/im2col.cuh:17-72) is an NHWC scatter that was never
// built; nothing is taken from it.
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <limits.h>

#include <type_traits>

#include "sd_common.h"
#include "sd_plan.cuh"

namespace sd {

struct ConvGeom {
    int N, C, H, W, R, S, P, Q;
    int pad_h, pad_w, stride_h, stride_w, dil_h, dil_w;
    int M, K;           // N*P*Q, C*R*S
    long long ldm;      // columns of colT that exist (>= M, multiple of 8)
    int Rb, Cb;         // plan grid: ceil(M/128) x ceil(K/128) (K as the GEMM sees it)
    long long kstride;  // elements from one k-row to the next: ldm, or 128 in the panel layout
    long long pstride;  // panel layout ([M/128][k_gemm][128], a kept block is one 32 KB run): elements per panel; else 0
};

// Offset of element (k, m) of the K-outer im2col matrix.  Eight consecutive m starting at a multiple of 8 are
// contiguous in either layout.
__device__ __forceinline__ long long col_off(const ConvGeom& g, long long k, long long m) {
    return g.pstride ? (m >> 7) * g.pstride + k * 128 + (m & 127) : k * g.ldm + m;
}

constexpr int kConvThreads = 256;

// Elements [e0, e0 + 8) of a row of `len` 16-bit elements, zero outside [0, len).  The row starts 16-byte aligned
// and len is a multiple of 8, so each of the (at most two) aligned 8-element chunks the window touches lies either
// entirely inside the row or entirely outside it: two 16-byte loads and a funnel shift replace eight 2-byte loads.
__device__ __forceinline__ void load8_shifted(const unsigned short* __restrict__ row, int e0, int len, uint32_t (&out)[4]) {
    const int a = e0 & ~7, sh = e0 - a;
    uint4 c0 = make_uint4(0, 0, 0, 0), c1 = make_uint4(0, 0, 0, 0);
    if (a >= 0 && a < len) c0 = __ldg(reinterpret_cast<const uint4*>(row + a));
    if (sh && a + 8 >= 0 && a + 8 < len) c1 = __ldg(reinterpret_cast<const uint4*>(row + a + 8));
    uint32_t w0 = c0.x, w1 = c0.y, w2 = c0.z, w3 = c0.w, w4 = c1.x, w5 = c1.y, w6 = c1.z, w7 = c1.w;
    const int ws = sh >> 1;
    if (ws & 1) { w0 = w1; w1 = w2; w2 = w3; w3 = w4; w4 = w5; w5 = w6; w6 = w7; }
    if (ws & 2) { w0 = w2; w1 = w3; w2 = w4; w3 = w5; w4 = w6; }
    const uint32_t sb = (sh & 1) * 16;
    out[0] = __funnelshift_r(w0, w1, sb);
    out[1] = __funnelshift_r(w1, w2, sb);
    out[2] = __funnelshift_r(w2, w3, sb);
    out[3] = __funnelshift_r(w3, w4, sb);
}

// Fast im2col for unit horizontal stride with W % 8 == 0 and Q % 8 == 0: the 8 output pixels a thread owns sit in
// one output row, so each k-row is one shifted 8-element window of one input row.
__global__ void __launch_bounds__(kConvThreads) im2col_kept_rows_kernel(const unsigned short* __restrict__ x,
                                                                        unsigned short* __restrict__ colT, ConvGeom g,
                                                                        const int* __restrict__ kept_pairs,
                                                                        const int* __restrict__ n_kept) {
    const int total = kept_pairs ? __ldg(n_kept) : g.Rb * g.Cb;
    const int mgrp = threadIdx.x & 15, ksub = threadIdx.x >> 4;
    const int PQ = g.P * g.Q, HW = g.H * g.W, RS = g.R * g.S;
    for (int t = blockIdx.x; t < total; t += gridDim.x) {
        const int mb = kept_pairs ? __ldg(kept_pairs + 2 * t) : t / g.Cb;
        const int kb = kept_pairs ? __ldg(kept_pairs + 2 * t + 1) : t - (t / g.Cb) * g.Cb;
        const int m0 = mb * 128 + mgrp * 8;
        if (m0 >= g.ldm) continue;
        const bool live = m0 < g.M;                      // M % 8 == 0 here, so the group is all in or all out
        const int n = live ? m0 / PQ : 0, pq = m0 - n * PQ, p = pq / g.Q, q0 = pq - p * g.Q;
        const unsigned short* xn = x + (long long)n * g.C * HW;
        const int hbase = p * g.stride_h - g.pad_h, wbase = q0 - g.pad_w;
        // (c, r*S + s) of this thread's first k-row; every pass advances k by 16 without dividing by C*R*S again
        int c = (kb * 128 + ksub) / RS, rs = (kb * 128 + ksub) - c * RS;
        const int c16 = 16 / RS, rs16 = 16 - c16 * RS;
#pragma unroll 2
        for (int pass = 0; pass < 8; ++pass) {
            const int k = kb * 128 + pass * 16 + ksub;
            if (k >= g.K) break;
            const int r = rs / g.S, s = rs - r * g.S;
            const int h = hbase + r * g.dil_h;
            uint32_t o[4] = {0, 0, 0, 0};
            if (live && (unsigned)h < (unsigned)g.H)
                load8_shifted(xn + (long long)c * HW + (long long)h * g.W, wbase + s * g.dil_w, g.W, o);
            *reinterpret_cast<uint4*>(colT + col_off(g, k, m0)) = make_uint4(o[0], o[1], o[2], o[3]);
            c += c16;
            rs += rs16;
            if (rs >= RS) { rs -= RS; ++c; }
        }
    }
}

// Fastest im2col: filters 3 wide with unit horizontal stride and dilation and one column of padding (so Q == W),
// rows of 8..128 pixels that divide 128.  The three taps s = 0, 1, 2 of one (c, r) read the same input row shifted
// by -1, 0, +1: a thread loads the aligned 8-pixel chunk once, borrows the one pixel on either side from its
// neighbour lanes (which own the neighbouring chunks of the same image row) and writes three k-rows.
__global__ void __launch_bounds__(kConvThreads) im2col_kept_s3_kernel(const unsigned short* __restrict__ x,
                                                                      unsigned short* __restrict__ colT, ConvGeom g,
                                                                      const int* __restrict__ kept_pairs,
                                                                      const int* __restrict__ n_kept) {
    const int total = kept_pairs ? __ldg(n_kept) : g.Rb * g.Cb;
    const int mgrp = threadIdx.x & 15, tsub = threadIdx.x >> 4;
    const int PQ = g.P * g.Q, HW = g.H * g.W;
    for (int t = blockIdx.x; t < total; t += gridDim.x) {
        const int mb = kept_pairs ? __ldg(kept_pairs + 2 * t) : t / g.Cb;
        const int kb = kept_pairs ? __ldg(kept_pairs + 2 * t + 1) : t - (t / g.Cb) * g.Cb;
        const int m0 = mb * 128 + mgrp * 8;
        const bool in_ld = m0 < g.ldm;                   // all lanes stay in the loop: they trade pixels below
        const bool live = m0 < g.M;                      // M % 8 == 0 here, so the group is all in or all out
        const int n = live ? m0 / PQ : 0, pq = m0 - n * PQ, p = pq / g.Q, q0 = pq - p * g.Q;
        const unsigned short* xn = x + (long long)n * g.C * HW;
        const int hbase = p * g.stride_h - g.pad_h;
        const bool has_left = q0 > 0, has_right = q0 + 8 < g.Q;
        const int k_lo = kb * 128, k_hi = min(k_lo + 128, g.K);
        // (c, r) pairs whose three k-rows 3 * (c * R + r) + s touch [k_lo, k_hi); the same number of passes for
        // every thread, because the shuffles below need whole warps
        const int cr_end = (k_hi + 2) / 3;
        for (int cr0 = k_lo / 3; cr0 < cr_end; cr0 += 16) {
            const int cr = cr0 + tsub;
            const bool valid = cr < cr_end;
            const int c = cr / g.R, r = cr - c * g.R;
            const int h = hbase + r * g.dil_h;
            uint4 v = make_uint4(0, 0, 0, 0);
            if (valid && live && (unsigned)h < (unsigned)g.H)
                v = __ldg(reinterpret_cast<const uint4*>(xn + (long long)c * HW + (long long)h * g.W + q0));
            uint32_t left = __shfl_up_sync(0xffffffffu, v.w, 1), right = __shfl_down_sync(0xffffffffu, v.x, 1);
            if (!has_left) left = 0;
            if (!has_right) right = 0;
            if (!valid || !in_ld) continue;
            const uint32_t a0 = __funnelshift_r(v.x, v.y, 16), a1 = __funnelshift_r(v.y, v.z, 16),
                           a2 = __funnelshift_r(v.z, v.w, 16);
            unsigned short* dst = colT + col_off(g, 3 * cr, m0);
            if (3 * cr >= k_lo)
                *reinterpret_cast<uint4*>(dst) = make_uint4(__funnelshift_r(left, v.x, 16), a0, a1, a2);
            if (3 * cr + 1 >= k_lo && 3 * cr + 1 < k_hi) *reinterpret_cast<uint4*>(dst + g.kstride) = v;
            if (3 * cr + 2 < k_hi)
                *reinterpret_cast<uint4*>(dst + 2 * g.kstride) = make_uint4(a0, a1, a2, __funnelshift_r(v.w, right, 16));
        }
    }
}

// One CTA per kept block (grid-stride): 128 k-rows x 128 m-columns of colT.  Thread t owns the 8 consecutive m
// starting at (t % 16) * 8 and visits k-rows (t / 16) + 16 * pass.  Bound by instruction issue, so the pixels are decoded by one
// division and counting on, and an element's address is the tap's pointer plus the pixel's offset (Off: 32 bits wherever
// eight images fit them).  64 x 64 x 56 x 56, 3x3 stride 2, 40 MB written: 25.7 us, 33.6 with a division per pixel and a
// 64-bit address per pixel and tap.
template <class Off>
__global__ void __launch_bounds__(kConvThreads) im2col_kept_kernel(const unsigned short* __restrict__ x,
                                                                   unsigned short* __restrict__ colT, ConvGeom g,
                                                                   const int* __restrict__ kept_pairs,
                                                                   const int* __restrict__ n_kept) {
    const int total = kept_pairs ? __ldg(n_kept) : g.Rb * g.Cb;
    const int mgrp = threadIdx.x & 15, ksub = threadIdx.x >> 4;
    const int PQ = g.P * g.Q, HW = g.H * g.W, RS = g.R * g.S;
    for (int t = blockIdx.x; t < total; t += gridDim.x) {
        const int mb = kept_pairs ? __ldg(kept_pairs + 2 * t) : t / g.Cb;
        const int kb = kept_pairs ? __ldg(kept_pairs + 2 * t + 1) : t - (t / g.Cb) * g.Cb;
        const int m0 = mb * 128 + mgrp * 8;
        if (m0 >= g.ldm) continue;
        const int n0 = m0 / PQ, pq0 = m0 - n0 * PQ;
        const unsigned short* image = x + (long long)n0 * g.C * HW;
        Off off[8];                       // of the pixel's tap (0, 0) in channel 0, from the first pixel's image
        int hb[8], wb[8];
        {
            int p = pq0 / g.Q, q = pq0 - p * g.Q;
            Off step = 0;
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                hb[j] = m0 + j < g.M ? p * g.stride_h - g.pad_h : -(1 << 28);   // never in range: padding columns are zero
                wb[j] = q * g.stride_w - g.pad_w;
                off[j] = step + Off(p * g.stride_h - g.pad_h) * g.W + wb[j];
                if (++q == g.Q) {
                    q = 0;
                    if (++p == g.P) { p = 0; step += Off(g.C) * HW; }
                }
            }
        }
#pragma unroll 2
        for (int pass = 0; pass < 8; ++pass) {
            const int k = kb * 128 + pass * 16 + ksub;
            if (k >= g.K) break;
            const int c = k / RS, rs = k - c * RS, r = rs / g.S, s = rs - r * g.S;
            const int hoff = r * g.dil_h, woff = s * g.dil_w;
            const unsigned short* tap = image + (long long)c * HW + (long long)hoff * g.W + woff;
            unsigned short v[8];
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const bool in = (unsigned)(hb[j] + hoff) < (unsigned)g.H && (unsigned)(wb[j] + woff) < (unsigned)g.W;
                v[j] = in ? __ldg(tap + off[j]) : (unsigned short)0;
            }
            uint4 o;
            o.x = v[0] | (uint32_t(v[1]) << 16);
            o.y = v[2] | (uint32_t(v[3]) << 16);
            o.z = v[4] | (uint32_t(v[5]) << 16);
            o.w = v[6] | (uint32_t(v[7]) << 16);
            *reinterpret_cast<uint4*>(colT + col_off(g, k, m0)) = o;
        }
    }
}

__device__ __forceinline__ float to_float(unsigned short v, int is_bf16) {
    return is_bf16 ? __bfloat162float(__ushort_as_bfloat16(v)) : __half2float(__ushort_as_half(v));
}
__device__ __forceinline__ unsigned short from_float(float f, int is_bf16) {
    return is_bf16 ? __bfloat16_as_ushort(__float2bfloat16_rn(f)) : __half_as_ushort(__float2half_rn(f));
}

// Eight consecutive results of dx starting at element 8 * i, as 16-bit values or in fp32 (an input kept in fp32 under
// autocast takes its gradient in fp32).
template <bool IS_BF16, bool OUT_F32>
__device__ __forceinline__ void store_dx8(void* dx, long long i, const float (&acc)[8]) {
    if (OUT_F32) {
        float4* d = static_cast<float4*>(dx) + 2 * i;
        d[0] = make_float4(acc[0], acc[1], acc[2], acc[3]);
        d[1] = make_float4(acc[4], acc[5], acc[6], acc[7]);
    } else {
        uint32_t out[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            if (IS_BF16) {
                __nv_bfloat162 v = __floats2bfloat162_rn(acc[2 * j], acc[2 * j + 1]);
                out[j] = *reinterpret_cast<uint32_t*>(&v);
            } else {
                __half2 v = __floats2half2_rn(acc[2 * j], acc[2 * j + 1]);
                out[j] = *reinterpret_cast<uint32_t*>(&v);
            }
        }
        static_cast<uint4*>(dx)[i] = make_uint4(out[0], out[1], out[2], out[3]);
    }
}

// col2im for any geometry, staged through shared memory.  A CTA owns a strip of SH input rows of CG channels of one image:
// it copies the CG x R x S runs of dcolT that feed them (each run is contiguous along m, read as aligned 16-byte chunks;
// chunks of dropped blocks become zeros) and then every thread gathers its results from there.  HBM-bound by design: each
// kept entry is read once, in full sectors.  Reading the taps straight from memory instead, two bytes per lane with a
// mask byte in front of every one, took 353 us on a 3x3 stride-2 layer (64 x 64 x 56 x 56) whose entries are 162 MB.
struct StripGeom {
    int SH, n_strips, CG, n_cgroups;
    int pitch;              // elements per run in shared memory
    int row_lanes;          // lanes that share one image row: a power of two, at most 32
    int sh_h;               // log2 of the vertical stride, or -1
};
__device__ __forceinline__ int div_stride(int v, int stride, int sh, bool* exact) {
    const int q = sh >= 0 ? v >> sh : v / stride;
    *exact = q * stride == v;
    return q;
}
template <bool IS_BF16, bool OUT_F32, int SMAX, int ST>
__global__ void __launch_bounds__(kConvThreads) col2im_kept_strip_kernel(const unsigned short* __restrict__ dcolT,
                                                                         void* __restrict__ dx, ConvGeom g, StripGeom sg,
                                                                         const unsigned char* __restrict__ tile_mask) {
    extern __shared__ __align__(16) unsigned short runs[];
    const int RS = g.R * g.S, PQ = g.P * g.Q;
    int u = blockIdx.x;
    const int strip = u % sg.n_strips;
    u /= sg.n_strips;
    const int c0 = (u % sg.n_cgroups) * sg.CG, n = u / sg.n_cgroups;
    const int cn = min(sg.CG, g.C - c0), h0 = strip * sg.SH, h1 = min(h0 + sg.SH, g.H);
    // output rows that any tap of the strip's input rows reads
    const int lo = h0 + g.pad_h - (g.R - 1) * g.dil_h, hi = h1 - 1 + g.pad_h;
    const int p0 = max(lo <= 0 ? 0 : (lo + g.stride_h - 1) / g.stride_h, 0), p1 = min(hi / g.stride_h + 1, g.P);
    const int m_first = n * PQ + p0 * g.Q, a0 = m_first & ~7;
    const int nch = p1 > p0 ? (n * PQ + p1 * g.Q - a0 + 7) >> 3 : 0;
    // four chunks of a thread at a time: their mask bytes, then their loads, are in flight together
    constexpr int LOADS = 4;
    for (int e0 = threadIdx.x; e0 < cn * RS * nch; e0 += LOADS * kConvThreads) {
        int k[LOADS], m[LOADS], at[LOADS];
        bool on[LOADS];
        uint4 v[LOADS];
#pragma unroll
        for (int j = 0; j < LOADS; ++j) {
            const int e = e0 + j * kConvThreads, row = e / nch, ch = e - row * nch;
            at[j] = e < cn * RS * nch ? row * sg.pitch + ch * 8 : -1;
            k[j] = c0 * RS + row;
            m[j] = a0 + ch * 8;
            on[j] = at[j] >= 0 && !(tile_mask && __ldg(tile_mask + (long long)(m[j] >> 7) * g.Cb + (k[j] >> 7)));
        }
#pragma unroll
        for (int j = 0; j < LOADS; ++j) {
            v[j] = make_uint4(0, 0, 0, 0);
            if (on[j]) v[j] = __ldg(reinterpret_cast<const uint4*>(dcolT + col_off(g, k[j], m[j])));
        }
#pragma unroll
        for (int j = 0; j < LOADS; ++j)
            if (at[j] >= 0) *reinterpret_cast<uint4*>(runs + at[j]) = v[j];
    }
    __syncthreads();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int rows_per_warp = 32 / sg.row_lanes, sub = lane / sg.row_lanes, wl = lane - sub * sg.row_lanes;
    const int base0 = n * PQ - a0;                                       // position of output pixel (0, 0) in a run
    // Under a horizontal stride of two (ST == 2) a thread gathers the results w = 2 j and 2 j + 1 of a row: tap s feeds exactly
    // one of them, the one of the parity of s * dil_w - pad_w, from q = j + const, and every lane has work at every tap.  Under
    // any other stride (ST == 1) it gathers one, and taps that miss it are skipped.
    const int J = (g.W + ST - 1) / ST;
    const bool whole_stores = ST == 2 && !(g.W & 1) && !(reinterpret_cast<uintptr_t>(dx) & 7);
    unsigned odd = 0;                                                    // ST == 2: taps that feed the second result
#pragma unroll
    for (int s = 0; s < SMAX; ++s)
        if (ST == 2 && ((s * g.dil_w - g.pad_w) & 1)) odd |= 1u << s;
    for (int j = wl; j < J; j += sg.row_lanes) {
        int q[SMAX];                                                     // where tap s reads in its run, or INT_MIN
#pragma unroll
        for (int s = 0; s < SMAX; ++s) {
            const int ww = ST * j + int(odd >> s & 1) + g.pad_w - s * g.dil_w;
            const int qq = ST == 2 ? ww >> 1 : g.stride_w == 1 ? ww : max(ww, 0) / g.stride_w;
            const bool exact = ST == 2 || qq * g.stride_w == ww;
            q[s] = (s < g.S && ww >= 0 && exact && qq < g.Q) ? s * sg.pitch + qq + base0 : INT_MIN;
        }
        // (channel, input row) pairs of this thread, without a division per pair
        const int rows = h1 - h0, step = (kConvThreads / 32) * rows_per_warp;
        int first = warp * rows_per_warp + sub, cg = first / rows, h = first - cg * rows;
        for (; cg < cn; h += step) {
            while (h >= rows) { h -= rows; ++cg; }
            if (cg >= cn) break;
            const unsigned short* src = runs + cg * RS * sg.pitch;
            const int top = h0 + h + g.pad_h;
            float acc[ST] = {};
            auto add_row = [&](const unsigned short* at) {
#pragma unroll
                for (int s = 0; s < SMAX; ++s)
                    if (q[s] != INT_MIN) {
                        const float f = to_float(at[q[s]], IS_BF16);
                        if (ST == 2 && (odd >> s & 1)) acc[ST - 1] += f; else acc[0] += f;
                    }
            };
            if (g.dil_h == 1) {
                // the filter rows that meet an output row: every stride_h-th one
                int r = sg.sh_h == 0 ? 0 : sg.sh_h > 0 ? top & (g.stride_h - 1) : top % g.stride_h;
                int p = sg.sh_h >= 0 ? (top - r) >> sg.sh_h : (top - r) / g.stride_h;
                if (p >= g.P) { r += (p - g.P + 1) * g.stride_h; p = g.P - 1; }
                for (; r < g.R && p >= 0; r += g.stride_h, --p) add_row(src + r * g.S * sg.pitch + p * g.Q);
            } else {
                for (int r = 0; r < g.R; ++r) {
                    const int hh = top - r * g.dil_h;
                    bool exact;
                    const int p = div_stride(max(hh, 0), g.stride_h, sg.sh_h, &exact);
                    if (hh < 0 || !exact || p >= g.P) continue;
                    add_row(src + r * g.S * sg.pitch + p * g.Q);
                }
            }
            const long long i = ((long long)(n * g.C + c0 + cg) * g.H + h0 + h) * g.W + ST * j;
            if (whole_stores) {                                          // both results in one store
                if (OUT_F32) *reinterpret_cast<float2*>(static_cast<float*>(dx) + i) = make_float2(acc[0], acc[ST - 1]);
                else *reinterpret_cast<uint32_t*>(static_cast<unsigned short*>(dx) + i) =
                         from_float(acc[0], IS_BF16) | (uint32_t(from_float(acc[ST - 1], IS_BF16)) << 16);
            } else {
#pragma unroll
                for (int b = 0; b < ST; ++b)
                    if (ST * j + b < g.W) {
                        if (OUT_F32) static_cast<float*>(dx)[i + b] = acc[b];
                        else static_cast<unsigned short*>(dx)[i + b] = from_float(acc[b], IS_BF16);
                    }
            }
        }
    }
}

// Adjoint of the kept-block im2col: dx[n,c,h,w] = sum over the filter taps (r,s) that map (h,w) to an output
// pixel (p,q) of dcolT[k(c,r,s)][m(n,p,q)], skipping dropped blocks (their entries are zero by definition).
// One thread per input element, consecutive threads along w.  Only for geometries whose strips do not fit shared memory
// (see col2im_kept_strip_kernel).
__global__ void __launch_bounds__(kConvThreads) col2im_kept_kernel(const unsigned short* __restrict__ dcolT,
                                                                   void* __restrict__ dx, ConvGeom g,
                                                                   const unsigned char* __restrict__ tile_mask,
                                                                   int is_bf16, int out_f32) {
    const long long total = (long long)g.N * g.C * g.H * g.W;
    const int PQ = g.P * g.Q, RS = g.R * g.S;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total;
         i += (long long)gridDim.x * blockDim.x) {
        const int w = int(i % g.W);
        long long rest = i / g.W;
        const int h = int(rest % g.H);
        rest /= g.H;
        const int c = int(rest % g.C), n = int(rest / g.C);
        float acc = 0.f;
        for (int r = 0; r < g.R; ++r) {
            const int hh = h + g.pad_h - r * g.dil_h;
            if (hh < 0 || hh % g.stride_h) continue;
            const int p = hh / g.stride_h;
            if (p >= g.P) continue;
            for (int s = 0; s < g.S; ++s) {
                const int ww = w + g.pad_w - s * g.dil_w;
                if (ww < 0 || ww % g.stride_w) continue;
                const int q = ww / g.stride_w;
                if (q >= g.Q) continue;
                const int m = n * PQ + p * g.Q + q, k = c * RS + r * g.S + s;
                if (tile_mask && tile_mask[(m >> 7) * g.Cb + (k >> 7)]) continue;
                acc += to_float(__ldg(dcolT + col_off(g, k, m)), is_bf16);
            }
        }
        if (out_f32) static_cast<float*>(dx)[i] = acc;
        else static_cast<unsigned short*>(dx)[i] = from_float(acc, is_bf16);
    }
}

// Fast col2im for unit strides with W % 8 == 0 and Q % 8 == 0: a thread owns 8 consecutive w of one (n, c, h);
// every filter tap is one shifted 8-element window of one dcolT row, whose aligned chunks each lie in one block.
template <bool IS_BF16, bool OUT_F32>
__global__ void __launch_bounds__(kConvThreads) col2im_kept_rows_kernel(const unsigned short* __restrict__ dcolT,
                                                                        void* __restrict__ dx, ConvGeom g,
                                                                        const unsigned char* __restrict__ tile_mask) {
    const int WG = g.W >> 3;
    const unsigned total = unsigned(g.N) * g.C * g.H * WG;       // the host checks that this fits 32 bits
    const int PQ = g.P * g.Q, RS = g.R * g.S;
    for (unsigned i = blockIdx.x * blockDim.x + threadIdx.x; i < total; i += gridDim.x * blockDim.x) {
        const int wg = int(i % WG);
        unsigned rest = i / WG;
        const int h = int(rest % g.H);
        rest /= g.H;
        const int c = int(rest % g.C), n = int(rest / g.C);
        float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
        for (int r = 0; r < g.R; ++r) {
            const int p = h + g.pad_h - r * g.dil_h;
            if ((unsigned)p >= (unsigned)g.P) continue;
            for (int s = 0; s < g.S; ++s) {
                const int k = c * RS + r * g.S + s;
                const int q0 = wg * 8 + g.pad_w - s * g.dil_w;        // output column that w = wg*8 fed through tap s
                const int a = q0 & ~7, sh = q0 - a;
                const long long mrow = (long long)n * PQ + (long long)p * g.Q;
                const unsigned short* rowa = dcolT + col_off(g, k, mrow + a);           // used only when the chunk exists
                const unsigned short* rowb = dcolT + col_off(g, k, mrow + a + 8);
                // chunk validity: inside [0, Q) and in a kept block
                uint4 c0 = make_uint4(0, 0, 0, 0), c1 = make_uint4(0, 0, 0, 0);
                if (a >= 0 && a < g.Q && !(tile_mask && tile_mask[((mrow + a) >> 7) * g.Cb + (k >> 7)]))
                    c0 = __ldg(reinterpret_cast<const uint4*>(rowa));
                if (sh && a + 8 >= 0 && a + 8 < g.Q && !(tile_mask && tile_mask[((mrow + a + 8) >> 7) * g.Cb + (k >> 7)]))
                    c1 = __ldg(reinterpret_cast<const uint4*>(rowb));
                uint32_t w0 = c0.x, w1 = c0.y, w2 = c0.z, w3 = c0.w, w4 = c1.x, w5 = c1.y, w6 = c1.z, w7 = c1.w;
                const int ws = sh >> 1;
                if (ws & 1) { w0 = w1; w1 = w2; w2 = w3; w3 = w4; w4 = w5; w5 = w6; w6 = w7; }
                if (ws & 2) { w0 = w2; w1 = w3; w2 = w4; w3 = w5; w4 = w6; }
                const uint32_t sb = (sh & 1) * 16;
                const uint32_t o[4] = {__funnelshift_r(w0, w1, sb), __funnelshift_r(w1, w2, sb),
                                       __funnelshift_r(w2, w3, sb), __funnelshift_r(w3, w4, sb)};
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    if (IS_BF16) {                               // bf16 -> fp32 is a 16-bit shift
                        acc[2 * j] += __uint_as_float(o[j] << 16);
                        acc[2 * j + 1] += __uint_as_float(o[j] & 0xffff0000u);
                    } else {
                        const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&o[j]));
                        acc[2 * j] += f.x;
                        acc[2 * j + 1] += f.y;
                    }
                }
            }
        }
        store_dx8<IS_BF16, OUT_F32>(dx, i, acc);
    }
}

// Fastest col2im: the adjoint of im2col_kept_s3_kernel under the same conditions plus unit vertical stride.  A thread
// owns 8 consecutive w of one (n, c, h) and reads, for each of the R x 3 taps, the aligned 8-pixel chunk of the tap's
// dcolT row; taps s = 0 and s = 2 are that chunk shifted by one pixel, the pixel that falls off going to the
// neighbour lane (which owns the neighbouring 8 pixels of the same image row).
template <bool IS_BF16, bool OUT_F32>
__global__ void __launch_bounds__(kConvThreads) col2im_kept_s3_kernel(const unsigned short* __restrict__ dcolT,
                                                                      void* __restrict__ dx, ConvGeom g,
                                                                      const unsigned char* __restrict__ tile_mask) {
    const int WG = g.W >> 3;                                     // lanes per image row; divides 32
    const unsigned total = unsigned(g.N) * g.C * g.H * WG;       // the host checks that this fits 32 bits
    const unsigned total_up = (total + 31u) & ~31u;              // whole warps run the loop: they trade pixels
    const int PQ = g.P * g.Q;
    for (unsigned i = blockIdx.x * blockDim.x + threadIdx.x; i < total_up; i += gridDim.x * blockDim.x) {
        const bool live = i < total;
        const int wg = int(i % WG);
        unsigned rest = i / WG;
        const int h = int(rest % g.H);
        rest /= g.H;
        const int c = live ? int(rest % g.C) : 0, n = live ? int(rest / g.C) : 0;
        const bool has_left = wg > 0, has_right = wg + 1 < WG;
        float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
        for (int r = 0; r < g.R; ++r) {
            const int p = h + g.pad_h - r * g.dil_h;
            const bool row_ok = live && (unsigned)p < (unsigned)g.P;
            const long long m = (long long)n * PQ + (long long)p * g.Q + wg * 8;
            const int k0 = (c * g.R + r) * 3;
            float f[3][8];
#pragma unroll
            for (int s = 0; s < 3; ++s) {
                const int k = k0 + s;
                uint4 v = make_uint4(0, 0, 0, 0);
                if (row_ok && !(tile_mask && tile_mask[(m >> 7) * g.Cb + (k >> 7)]))
                    v = __ldg(reinterpret_cast<const uint4*>(dcolT + col_off(g, k, m)));
                const uint32_t wv[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    if (IS_BF16) {                               // bf16 -> fp32 is a 16-bit shift
                        f[s][2 * j] = __uint_as_float(wv[j] << 16);
                        f[s][2 * j + 1] = __uint_as_float(wv[j] & 0xffff0000u);
                    } else {
                        const float2 t = __half22float2(*reinterpret_cast<const __half2*>(&wv[j]));
                        f[s][2 * j] = t.x;
                        f[s][2 * j + 1] = t.y;
                    }
                }
            }
            // dx[w] += dcol[s][q = w + 1 - s]: tap 0 reads one pixel to the right, tap 2 one to the left
            float from_right = __shfl_down_sync(0xffffffffu, f[0][0], 1);
            float from_left = __shfl_up_sync(0xffffffffu, f[2][7], 1);
            if (!has_right) from_right = 0.f;
            if (!has_left) from_left = 0.f;
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                acc[j] += f[1][j];
                acc[j] += j < 7 ? f[0][j + 1] : from_right;
                acc[j] += j > 0 ? f[2][j - 1] : from_left;
            }
        }
        if (!live) continue;
        store_dx8<IS_BF16, OUT_F32>(dx, i, acc);
    }
}

// The same for 3 x 3 filters, unrolled over all nine taps: first the nine block-mask bytes, then the nine chunk loads
// (independent of one another, so one memory round trip covers them all), then the arithmetic.
template <bool IS_BF16, bool OUT_F32>
__global__ void __launch_bounds__(kConvThreads) col2im_kept_3x3_kernel(const unsigned short* __restrict__ dcolT,
                                                                       void* __restrict__ dx, ConvGeom g,
                                                                       const unsigned char* __restrict__ tile_mask) {
    const int WG = g.W >> 3, wg_bits = 31 - __clz(WG);           // lanes per image row: a power of two up to 16
    const unsigned total = unsigned(g.N) * g.C * g.H * WG;       // the host checks that this fits 32 bits
    const unsigned total_up = (total + 31u) & ~31u;              // whole warps run the loop: they trade pixels
    const int PQ = g.P * g.Q;
    const long long tap_step = g.kstride;
    for (unsigned i = blockIdx.x * blockDim.x + threadIdx.x; i < total_up; i += gridDim.x * blockDim.x) {
        const bool live = i < total;
        const int wg = int(i & (WG - 1));
        unsigned rest = i >> wg_bits;
        const int h = int(rest % g.H);
        rest /= g.H;
        const int c = live ? int(rest % g.C) : 0, n = live ? int(rest / g.C) : 0;
        const int p0 = h + g.pad_h, k0 = c * 9;
        const long long m0 = (long long)n * PQ + wg * 8;
        const unsigned short* src[3];                             // tap (r, 0) of each filter row
        bool ok[9];
#pragma unroll
        for (int r = 0; r < 3; ++r) {
            const int p = p0 - r * g.dil_h;
            const bool row_ok = live && (unsigned)p < (unsigned)g.P;
            const long long m = m0 + (long long)p * g.Q;
            src[r] = dcolT + col_off(g, k0 + 3 * r, m);
            const int mrow = int(m >> 7) * g.Cb;
#pragma unroll
            for (int s = 0; s < 3; ++s)
                ok[3 * r + s] = row_ok && !(tile_mask && __ldg(tile_mask + mrow + ((k0 + 3 * r + s) >> 7)));
        }
        uint4 v[9];
#pragma unroll
        for (int r = 0; r < 3; ++r)
#pragma unroll
            for (int s = 0; s < 3; ++s)
                v[3 * r + s] = ok[3 * r + s] ? __ldg(reinterpret_cast<const uint4*>(src[r] + s * tap_step))
                                             : make_uint4(0, 0, 0, 0);
        const bool has_left = wg > 0, has_right = wg + 1 < WG;
        float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int r = 0; r < 3; ++r) {
            float f[3][8];
#pragma unroll
            for (int s = 0; s < 3; ++s) {
                const uint32_t wv[4] = {v[3 * r + s].x, v[3 * r + s].y, v[3 * r + s].z, v[3 * r + s].w};
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    if (IS_BF16) {                               // bf16 -> fp32 is a 16-bit shift
                        f[s][2 * j] = __uint_as_float(wv[j] << 16);
                        f[s][2 * j + 1] = __uint_as_float(wv[j] & 0xffff0000u);
                    } else {
                        const float2 t = __half22float2(*reinterpret_cast<const __half2*>(&wv[j]));
                        f[s][2 * j] = t.x;
                        f[s][2 * j + 1] = t.y;
                    }
                }
            }
            // dx[w] += dcol[s][q = w + 1 - s]: tap 0 reads one pixel to the right, tap 2 one to the left
            float from_right = __shfl_down_sync(0xffffffffu, f[0][0], 1);
            float from_left = __shfl_up_sync(0xffffffffu, f[2][7], 1);
            if (!has_right) from_right = 0.f;
            if (!has_left) from_left = 0.f;
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                acc[j] += f[1][j];
                acc[j] += j < 7 ? f[0][j + 1] : from_right;
                acc[j] += j > 0 ? f[2][j - 1] : from_left;
            }
        }
        if (!live) continue;
        store_dx8<IS_BF16, OUT_F32>(dx, i, acc);
    }
}

static int make_geom(ConvGeom* g, int N, int C, int H, int W, int R, int S, int pad_h, int pad_w, int stride_h,
                     int stride_w, int dil_h, int dil_w, int64_t ldm, int k_gemm, bool panels = false) {
    if (N <= 0 || C <= 0 || H <= 0 || W <= 0 || R <= 0 || S <= 0)
        return fail(SD_ERR_INVALID_ARG, "conv sizes must be positive");
    if (stride_h <= 0 || stride_w <= 0 || dil_h <= 0 || dil_w <= 0 || pad_h < 0 || pad_w < 0)
        return fail(SD_ERR_INVALID_ARG, "stride and dilation must be positive, padding non-negative");
    const long long over_h = H + 2ll * pad_h - (long long)dil_h * (R - 1) - 1;   // rows and columns the filter can move over
    const long long over_w = W + 2ll * pad_w - (long long)dil_w * (S - 1) - 1;
    if (over_h < 0 || over_w < 0) return fail(SD_ERR_INVALID_ARG, "the filter does not fit the padded input");
    const long long P = over_h / stride_h + 1, Q = over_w / stride_w + 1;
    const long long M = N * P * Q, K = (long long)C * R * S;
    if (M > (1ll << 30) || K > (1ll << 30)) return fail(SD_ERR_TOO_LARGE, "im2col matrix too large (M=%lld, K=%lld)", M, K);
    if (panels) ldm = ((M + 127) / 128) * 128;      // whole panels exist
    if (ldm < M || (ldm & 7)) return fail(SD_ERR_LAYOUT, "ldm (%lld) must be >= N*P*Q (%lld) and a multiple of 8", (long long)ldm, M);
    if (k_gemm < K) return fail(SD_ERR_INVALID_ARG, "k_gemm (%d) must be >= C*R*S (%lld)", k_gemm, K);
    *g = ConvGeom{N, C, H, W, R, S, int(P), int(Q), pad_h, pad_w, stride_h, stride_w, dil_h, dil_w, int(M), int(K), ldm,
                  int((M + 127) / 128), (k_gemm + 127) / 128, panels ? 128 : ldm, panels ? (long long)k_gemm * 128 : 0};
    return SD_OK;
}

// Strip height and channels per CTA of the staged col2im, and its shared memory; false if the geometry does not fit.
// Strips are as tall as 40 KB of runs allow (the overlap of neighbouring strips is read twice); small images take several
// channels per CTA, so that a CTA has at least about a thousand results to gather.
static bool strip_geom(const ConvGeom& g, uintptr_t src, StripGeom* sg, int* bytes) {
    if (g.S > 7 || (src & 15)) return false;
    const int RS = g.R * g.S;
    auto run_elems = [&](int SH) {
        long long np = (SH - 1 + (long long)(g.R - 1) * g.dil_h) / g.stride_h + 2;
        if (np > g.P) np = g.P;
        return ((np * g.Q + 14) & ~7ll) + 8;                  // start and end rounded to chunks of 8
    };
    int SH = g.H;
    while (SH > 1 && run_elems(SH) * RS * 2 > 40 * 1024) SH = (SH + 1) / 2;
    const long long one = run_elems(SH) * RS * 2;
    if (one > 44 * 1024) return false;
    int CG = 1;
    while (CG * 2 <= g.C && one * CG * 2 <= 24 * 1024 && (long long)CG * SH * g.W < 1024) CG *= 2;
    sg->SH = SH;
    sg->n_strips = (g.H + SH - 1) / SH;
    sg->CG = CG;
    sg->n_cgroups = (g.C + CG - 1) / CG;
    sg->pitch = int(run_elems(SH));
    sg->row_lanes = 1;
    while (sg->row_lanes * (g.stride_w == 2 ? 2 : 1) < g.W && sg->row_lanes < 32) sg->row_lanes *= 2;
    auto log2_or = [](int v) { int l = 0; while ((1 << l) < v) ++l; return (1 << l) == v ? l : -1; };
    sg->sh_h = log2_or(g.stride_h);
    if ((long long)g.N * sg->n_cgroups * sg->n_strips > (1ll << 31) - 1) return false;
    *bytes = int(one * CG);
    return true;
}

}  // namespace sd

static int im2col_kept_impl(const void* x, int N, int C, int H, int W, int R, int S, int pad_h, int pad_w, int stride_h,
                            int stride_w, int dil_h, int dil_w, void* colT, int64_t ldm, int k_gemm, const void* plan,
                            void* stream, bool panels) {
    if (!x || !colT) return sd::fail(SD_ERR_INVALID_ARG, "x or colT is null");
    if ((reinterpret_cast<uintptr_t>(colT) & 15)) return sd::fail(SD_ERR_LAYOUT, "colT must be 16-byte aligned");
    sd::ConvGeom g;
    int rc = sd::make_geom(&g, N, C, H, W, R, S, pad_h, pad_w, stride_h, stride_w, dil_h, dil_w, ldm, k_gemm, panels);
    if (rc) return rc;
    const int *pairs = nullptr, *n_kept = nullptr;
    if (plan) {
        const sd_plan_layout L = sd::plan_layout(g.Rb, g.Cb);
        const unsigned char* b = static_cast<const unsigned char*>(plan);
        pairs = reinterpret_cast<const int*>(b + L.kept_pairs);
        n_kept = reinterpret_cast<const int*>(b + L.header) + sd::H_NNZ;
    }
    int sms = 0;
    rc = sd::sm_count_current_device(&sms);
    if (rc) return rc;
    long long blocks = (long long)g.Rb * g.Cb;
    int grid = int(blocks < (long long)sms * 8 ? blocks : (long long)sms * 8);
    const bool rows_path = stride_w == 1 && (W & 7) == 0 && (g.Q & 7) == 0 && (reinterpret_cast<uintptr_t>(x) & 15) == 0;
    const bool s3_path = rows_path && S == 3 && dil_w == 1 && pad_w == 1 && W <= 128 && 128 % W == 0;
    if (s3_path)
        sd::im2col_kept_s3_kernel<<<grid, sd::kConvThreads, 0, static_cast<cudaStream_t>(stream)>>>(
            static_cast<const unsigned short*>(x), static_cast<unsigned short*>(colT), g, pairs, n_kept);
    else if (rows_path)
        sd::im2col_kept_rows_kernel<<<grid, sd::kConvThreads, 0, static_cast<cudaStream_t>(stream)>>>(
            static_cast<const unsigned short*>(x), static_cast<unsigned short*>(colT), g, pairs, n_kept);
    else {
        // offsets span at most nine images and the padding around them
        const bool small = (long long)C * H * W < (1ll << 27) && (long long)(pad_h + 1) * W < (1ll << 27) && pad_w < (1 << 27);
        auto kernel = small ? &sd::im2col_kept_kernel<int> : &sd::im2col_kept_kernel<long long>;
        kernel<<<grid, sd::kConvThreads, 0, static_cast<cudaStream_t>(stream)>>>(
            static_cast<const unsigned short*>(x), static_cast<unsigned short*>(colT), g, pairs, n_kept);
    }
    SD_CUDA_TRY(cudaGetLastError());
    return SD_OK;
}

static int col2im_kept_impl(const void* dcolT, int64_t ldm, int k_gemm, int N, int C, int H, int W, int R, int S, int pad_h,
                            int pad_w, int stride_h, int stride_w, int dil_h, int dil_w, void* dx, const void* plan,
                            int dtype, void* stream, bool panels, bool out_f32 = false) {
    if (!dcolT || !dx) return sd::fail(SD_ERR_INVALID_ARG, "dcolT or dx is null");
    if (dtype != SD_F16 && dtype != SD_BF16) return sd::fail(SD_ERR_INVALID_ARG, "dtype must be SD_F16 or SD_BF16");
    sd::ConvGeom g;
    int rc = sd::make_geom(&g, N, C, H, W, R, S, pad_h, pad_w, stride_h, stride_w, dil_h, dil_w, ldm, k_gemm, panels);
    if (rc) return rc;
    const unsigned char* mask = nullptr;
    if (plan) mask = static_cast<const unsigned char*>(plan) + sd::plan_layout(g.Rb, g.Cb).mask;
    int sms = 0;
    rc = sd::sm_count_current_device(&sms);
    if (rc) return rc;
    const bool rows_path = stride_w == 1 && stride_h == 1 && (W & 7) == 0 && (g.Q & 7) == 0 &&
                           ((reinterpret_cast<uintptr_t>(dcolT) | reinterpret_cast<uintptr_t>(dx)) & 15) == 0 &&
                           (long long)N * C * H * (W / 8) < (1ll << 31);
    const long long total = (long long)N * C * H * (rows_path ? W / 8 : W);
    long long blocks = (total + sd::kConvThreads - 1) / sd::kConvThreads;
    int grid = int(blocks < (long long)sms * 16 ? blocks : (long long)sms * 16);
    const bool s3_path = rows_path && S == 3 && dil_w == 1 && pad_w == 1 && W <= 128 && 128 % W == 0;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const unsigned short* src = static_cast<const unsigned short*>(dcolT);
    auto by_type = [&](auto&& launch) {                      // launch(bf16, fp32 result) as compile-time flags
        if (dtype == SD_BF16) {
            if (out_f32) launch(std::true_type{}, std::true_type{}); else launch(std::true_type{}, std::false_type{});
        } else {
            if (out_f32) launch(std::false_type{}, std::true_type{}); else launch(std::false_type{}, std::false_type{});
        }
    };
    sd::StripGeom sg;
    int strip_bytes = 0;
    if (s3_path && R == 3)
        by_type([&](auto bf, auto f32) { sd::col2im_kept_3x3_kernel<bf.value, f32.value><<<grid, sd::kConvThreads, 0, st>>>(src, dx, g, mask); });
    else if (s3_path)
        by_type([&](auto bf, auto f32) { sd::col2im_kept_s3_kernel<bf.value, f32.value><<<grid, sd::kConvThreads, 0, st>>>(src, dx, g, mask); });
    else if (rows_path)
        by_type([&](auto bf, auto f32) { sd::col2im_kept_rows_kernel<bf.value, f32.value><<<grid, sd::kConvThreads, 0, st>>>(src, dx, g, mask); });
    else if (sd::strip_geom(g, reinterpret_cast<uintptr_t>(dcolT), &sg, &strip_bytes)) {
        const unsigned n_cta = unsigned(N) * sg.n_cgroups * sg.n_strips;
        by_type([&](auto bf, auto f32) {
            auto kernel = S <= 3 ? (stride_w != 2 ? &sd::col2im_kept_strip_kernel<bf.value, f32.value, 3, 1> : &sd::col2im_kept_strip_kernel<bf.value, f32.value, 3, 2>)
                                 : (stride_w != 2 ? &sd::col2im_kept_strip_kernel<bf.value, f32.value, 7, 1> : &sd::col2im_kept_strip_kernel<bf.value, f32.value, 7, 2>);
            kernel<<<n_cta, sd::kConvThreads, strip_bytes, st>>>(src, dx, g, sg, mask);
        });
    } else
        sd::col2im_kept_kernel<<<grid, sd::kConvThreads, 0, st>>>(src, dx, g, mask, dtype == SD_BF16, out_f32);
    SD_CUDA_TRY(cudaGetLastError());
    return SD_OK;
}

extern "C" {

int sd_im2col_kept(const void* x, int N, int C, int H, int W, int R, int S, int pad_h, int pad_w, int stride_h,
                   int stride_w, int dil_h, int dil_w, void* colT, int64_t ldm, int k_gemm, const void* plan,
                   void* stream) {
    return im2col_kept_impl(x, N, C, H, W, R, S, pad_h, pad_w, stride_h, stride_w, dil_h, dil_w, colT, ldm, k_gemm, plan,
                            stream, false);
}

int sd_im2col_kept_panels(const void* x, int N, int C, int H, int W, int R, int S, int pad_h, int pad_w, int stride_h,
                          int stride_w, int dil_h, int dil_w, void* col_panels, int k_gemm, const void* plan,
                          void* stream) {
    return im2col_kept_impl(x, N, C, H, W, R, S, pad_h, pad_w, stride_h, stride_w, dil_h, dil_w, col_panels, 0, k_gemm,
                            plan, stream, true);
}

int sd_col2im_kept(const void* dcolT, int64_t ldm, int k_gemm, int N, int C, int H, int W, int R, int S, int pad_h,
                   int pad_w, int stride_h, int stride_w, int dil_h, int dil_w, void* dx, const void* plan, int dtype,
                   void* stream) {
    return col2im_kept_impl(dcolT, ldm, k_gemm, N, C, H, W, R, S, pad_h, pad_w, stride_h, stride_w, dil_h, dil_w, dx,
                            plan, dtype, stream, false);
}

int sd_col2im_kept_panels_f32(const void* dcol_panels, int k_gemm, int N, int C, int H, int W, int R, int S, int pad_h,
                              int pad_w, int stride_h, int stride_w, int dil_h, int dil_w, float* dx, const void* plan,
                              int dtype, void* stream) {
    return col2im_kept_impl(dcol_panels, 0, k_gemm, N, C, H, W, R, S, pad_h, pad_w, stride_h, stride_w, dil_h, dil_w,
                            dx, plan, dtype, stream, true, true);
}

int sd_col2im_kept_panels(const void* dcol_panels, int k_gemm, int N, int C, int H, int W, int R, int S, int pad_h,
                          int pad_w, int stride_h, int stride_w, int dil_h, int dil_w, void* dx, const void* plan,
                          int dtype, void* stream) {
    return col2im_kept_impl(dcol_panels, 0, k_gemm, N, C, H, W, R, S, pad_h, pad_w, stride_h, stride_w, dil_h, dil_w,
                            dx, plan, dtype, stream, true);
}

}  // extern "C"
