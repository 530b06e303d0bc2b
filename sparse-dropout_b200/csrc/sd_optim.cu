// AdamW over all parameters of a model in one launch.
//
// The reference trains with torch.optim.AdamW(fused=True) (eval/llm/model.py:157-173).  torch's multi-tensor kernel hands out
// chunks of 65 536 elements, 46 CTAs for the 3 M parameters of the MLP, and a separate launch adds one to every step
// counter: 67 us where the 28 bytes per parameter take 13 us of HBM time (less when they still sit in L2).  Here a CTA takes
// kAdamChunk elements of one tensor, so a model of a few million parameters fills the GPU; the last CTA to finish advances the
// step counters.
#include "sd_common.h"

namespace sd {

constexpr int kAdamThreads = 256;
constexpr int kAdamChunk = SD_ADAMW_CHUNK;
static_assert(kAdamChunk == kAdamThreads * 8, "two float4 groups per thread");

struct AdamTable {                                // device memory: this header, then entries, then chunks
    int done, n_tensors, n_chunks, pad;
};
struct AdamHyper {
    double lr[SD_ADAMW_MAX_GROUPS], beta1[SD_ADAMW_MAX_GROUPS], beta2[SD_ADAMW_MAX_GROUPS], eps[SD_ADAMW_MAX_GROUPS],
        weight_decay[SD_ADAMW_MAX_GROUPS];
};

// The second moment is computed in double and rounded once, as torch does: in fp32 the rounding of beta2 alone is half an ulp
// of the result, and its error was 1.2 times torch's.
struct AdamStep {
    double b2, one_minus_b2;
    float decay, one_minus_b1, step_size, inv_bias2_sqrt, eps;
    __device__ __forceinline__ void apply(float& p, float g, float& m, float& v) const {
        p *= decay;
        m += (g - m) * one_minus_b1;
        v = float(b2 * double(v) + one_minus_b2 * double(g) * double(g));
        p -= step_size * m / (sqrtf(v) * inv_bias2_sqrt + eps);
    }
};

__global__ void __launch_bounds__(kAdamThreads) adamw_kernel(AdamTable* table, AdamHyper h) {
    const sd_adamw_entry* entries = reinterpret_cast<const sd_adamw_entry*>(table + 1);
    const int2 chunk = reinterpret_cast<const int2*>(entries + table->n_tensors)[blockIdx.x];
    const sd_adamw_entry e = entries[chunk.x];
    __shared__ AdamStep st;
    if (threadIdx.x == 0) {
        const double t = double(*e.step) + 1.0;   // every CTA reads the counter before the last one advances it
        const double lr = h.lr[e.group], b1 = h.beta1[e.group], b2 = h.beta2[e.group];
        st.decay = float(1.0 - lr * h.weight_decay[e.group]);
        st.one_minus_b1 = float(1.0 - b1);
        st.b2 = b2;
        st.one_minus_b2 = 1.0 - b2;
        st.step_size = float(lr / (1.0 - pow(b1, t)));
        st.inv_bias2_sqrt = float(1.0 / sqrt(1.0 - pow(b2, t)));
        st.eps = float(h.eps[e.group]);
    }
    const long long base = (long long)chunk.y * kAdamChunk;
    // loads before the barrier: they do not depend on the step's constants
    float4 p[2], g[2], m[2], v[2];
    long long at[2];
    int full[2];
#pragma unroll
    for (int j = 0; j < 2; ++j) {
        at[j] = base + (j * kAdamThreads + threadIdx.x) * 4;
        full[j] = at[j] + 4 <= e.n;
        if (full[j]) {
            p[j] = *reinterpret_cast<const float4*>(e.p + at[j]);
            g[j] = __ldg(reinterpret_cast<const float4*>(e.g + at[j]));
            m[j] = *reinterpret_cast<const float4*>(e.m + at[j]);
            v[j] = *reinterpret_cast<const float4*>(e.v + at[j]);
        }
    }
    __syncthreads();
    const AdamStep s = st;
#pragma unroll
    for (int j = 0; j < 2; ++j) {
        if (full[j]) {
            s.apply(p[j].x, g[j].x, m[j].x, v[j].x);
            s.apply(p[j].y, g[j].y, m[j].y, v[j].y);
            s.apply(p[j].z, g[j].z, m[j].z, v[j].z);
            s.apply(p[j].w, g[j].w, m[j].w, v[j].w);
            *reinterpret_cast<float4*>(e.p + at[j]) = p[j];
            *reinterpret_cast<float4*>(e.m + at[j]) = m[j];
            *reinterpret_cast<float4*>(e.v + at[j]) = v[j];
        } else {
            for (long long i = at[j]; i < e.n && i < at[j] + 4; ++i) {
                float pp = e.p[i], mm = e.m[i], vv = e.v[i];
                s.apply(pp, e.g[i], mm, vv);
                e.p[i] = pp;
                e.m[i] = mm;
                e.v[i] = vv;
            }
        }
    }
    __shared__ int last;
    if (threadIdx.x == 0) last = atomicAdd(&table->done, 1) == int(gridDim.x) - 1;
    __syncthreads();
    if (last) {
        for (int i = threadIdx.x; i < table->n_tensors; i += kAdamThreads) *entries[i].step += 1.f;
        if (threadIdx.x == 0) table->done = 0;
    }
}

}  // namespace sd

extern "C" {

static long long adamw_chunks(const sd_adamw_entry* e, int n) {
    long long c = 0;
    for (int i = 0; i < n; ++i) c += (e[i].n + sd::kAdamChunk - 1) / sd::kAdamChunk;
    return c;
}

size_t sd_adamw_table_bytes(const sd_adamw_entry* entries, int n) {
    if (!entries || n <= 0) return 0;
    return sizeof(sd::AdamTable) + size_t(n) * sizeof(sd_adamw_entry) + size_t(adamw_chunks(entries, n)) * sizeof(int2);
}

int sd_adamw_table_fill(void* host_table, const sd_adamw_entry* entries, int n) {
    if (!host_table || !entries || n <= 0) return sd::fail(SD_ERR_INVALID_ARG, "sd_adamw_table_fill: bad arguments");
    for (int i = 0; i < n; ++i) {
        const sd_adamw_entry& e = entries[i];
        if (!e.p || !e.g || !e.m || !e.v || !e.step || e.n <= 0 || e.group < 0 || e.group >= SD_ADAMW_MAX_GROUPS)
            return sd::fail(SD_ERR_INVALID_ARG, "sd_adamw_table_fill: entry %d is incomplete", i);
        if ((reinterpret_cast<uintptr_t>(e.p) | reinterpret_cast<uintptr_t>(e.g) | reinterpret_cast<uintptr_t>(e.m) |
             reinterpret_cast<uintptr_t>(e.v)) & 15)
            return sd::fail(SD_ERR_LAYOUT, "sd_adamw_table_fill: entry %d is not 16-byte aligned", i);
    }
    const long long chunks = adamw_chunks(entries, n);
    if (chunks > (1ll << 30)) return sd::fail(SD_ERR_TOO_LARGE, "sd_adamw_table_fill: too many elements");
    auto* t = static_cast<sd::AdamTable*>(host_table);
    *t = sd::AdamTable{0, n, int(chunks), 0};
    auto* dst = reinterpret_cast<sd_adamw_entry*>(t + 1);
    auto* c = reinterpret_cast<int2*>(dst + n);
    for (int i = 0; i < n; ++i) {
        dst[i] = entries[i];
        const int k = int((entries[i].n + sd::kAdamChunk - 1) / sd::kAdamChunk);
        for (int j = 0; j < k; ++j) *c++ = make_int2(i, j);
    }
    return SD_OK;
}

int sd_adamw_step(void* device_table, int64_t n_chunks, const double* hyper, int n_groups, void* stream) {
    if (!device_table || !hyper || n_chunks <= 0 || n_chunks > (1ll << 30) || n_groups <= 0 || n_groups > SD_ADAMW_MAX_GROUPS)
        return sd::fail(SD_ERR_INVALID_ARG, "sd_adamw_step: bad arguments");
    sd::AdamHyper h{};
    for (int i = 0; i < n_groups; ++i) {
        h.lr[i] = hyper[5 * i];
        h.beta1[i] = hyper[5 * i + 1];
        h.beta2[i] = hyper[5 * i + 2];
        h.eps[i] = hyper[5 * i + 3];
        h.weight_decay[i] = hyper[5 * i + 4];
    }
    sd::adamw_kernel<<<int(n_chunks), sd::kAdamThreads, 0, static_cast<cudaStream_t>(stream)>>>(static_cast<sd::AdamTable*>(device_table), h);
    SD_CUDA_TRY(cudaGetLastError());
    return SD_OK;
}

}  // extern "C"
