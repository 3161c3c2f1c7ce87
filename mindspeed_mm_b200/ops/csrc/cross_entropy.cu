// Row-wise softmax cross entropy that turns bf16 logits into their gradient in place.
//
//   loss[t]   = logsumexp(z[t, :]) - z[t, label[t]]           (0 for ignored rows)
//   z[t, :]  <- (softmax(z[t, :]) - onehot(label[t]))          (0 for ignored rows)
//
// Rows without a target take no part: the rows with one are listed first (label_rows_kernel), and the products and this kernel run over
// them alone.
//
// One CTA per row, two passes: pass 1 keeps a running (max, sum) per thread (online softmax) and merges
// them across the block; pass 2 re-reads the row (304 KB for V = 152064: still L2-resident) and writes
// the gradient.  fp32 math on bf16 storage; V must be a multiple of 8 and rows 16-byte aligned.
#include "common.cuh"

namespace {

constexpr int kCEThreads = 512;

__global__ void __launch_bounds__(kCEThreads) ce_fwd_bwd_kernel(bf16* __restrict__ z, long long ld,
                                                                const long long* __restrict__ labels,
                                                                float* __restrict__ loss, int V, int ignore_index,
                                                                const int* __restrict__ src, const int* __restrict__ count, int base) {
    let_successor_start();
    __shared__ float red[72];
    const long long row = blockIdx.x;
    Vec8* zr = reinterpret_cast<Vec8*>(z + row * ld);
    const int nvec = V >> 3;
    // src: row `base + row` of the list stands for token src[base + row]; `count` of them are in use.  The rows up to the next multiple of 64
    // are zeros (the weight's gradient reads them), what lies behind is not touched.
    if (src != nullptr && row >= ((max(0, *count - base) + 63) & ~63)) {
        if (threadIdx.x == 0) loss[row] = 0.f;
        return;
    }
    const int token = src == nullptr ? (int)row : src[base + row];
    const long long label = token < 0 ? ignore_index : labels[token];
    if (label == ignore_index) {
        Vec8 zero;
#pragma unroll
        for (int i = 0; i < 4; ++i) zero.v[i] = __floats2bfloat162_rn(0.f, 0.f);
        for (int i = threadIdx.x; i < nvec; i += kCEThreads) zr[i] = zero;
        if (threadIdx.x == 0) loss[row] = 0.f;
        return;
    }
    float m = -INFINITY, s = 0.f;
    for (int i = threadIdx.x; i < nvec; i += kCEThreads) {
        float f[8];
        unpack8(zr[i], f);
        float lm = f[0];
#pragma unroll
        for (int k = 1; k < 8; ++k) lm = fmaxf(lm, f[k]);
        const float nm = fmaxf(m, lm);
        float acc = 0.f;
#pragma unroll
        for (int k = 0; k < 8; ++k) acc += __expf(f[k] - nm);
        s = s * __expf(m - nm) + acc;
        m = nm;
    }
    // block max
    float wm = warp_max(m);
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    if (lane == 0) red[wid] = wm;
    __syncthreads();
    float M = red[lane < (kCEThreads >> 5) ? lane : 0];
    M = warp_max(M);
    __syncthreads();
    const float S = block_sum(s * __expf(m - M), red);
    const float lse = M + __logf(S);
    if (threadIdx.x == 0) loss[row] = lse - __bfloat162float(z[row * ld + label]);
    __syncthreads();  // the label logit has been read before anyone overwrites it
    const int lvec = (int)(label >> 3), lpos = (int)(label & 7);
    for (int i = threadIdx.x; i < nvec; i += kCEThreads) {
        float f[8];
        unpack8(zr[i], f);
#pragma unroll
        for (int k = 0; k < 8; ++k) f[k] = __expf(f[k] - lse);
        if (i == lvec) f[lpos] -= 1.f;
        zr[i] = pack8(f);
    }
}

// Rows with a target, in their order: src[i] = token of the i-th, row[t] = its place (-1: none), *count of them; src is -1 behind them.
// One block, eight labels a thread and step: 8192 labels in 4 us.
constexpr int kListThreads = 1024, kListEach = 8;
__global__ void __launch_bounds__(kListThreads) label_rows_kernel(const long long* __restrict__ labels, int T, int ignore_index,
                                                                 int* __restrict__ src, int* __restrict__ row, int* __restrict__ count) {
    let_successor_start();
    __shared__ int sums[32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    int base = 0;
    for (int t0 = 0; t0 < T; t0 += kListThreads * kListEach) {
        const int first = t0 + threadIdx.x * kListEach;
        unsigned used = 0;
#pragma unroll
        for (int i = 0; i < kListEach; ++i)
            if (first + i < T && labels[first + i] != ignore_index) used |= 1u << i;
        int upto = __popc(used);
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int v = __shfl_up_sync(0xffffffffu, upto, o);
            if (lane >= o) upto += v;
        }
        if (lane == 31) sums[w] = upto;
        __syncthreads();
        int total = 0;
        for (int i = 0; i < kListThreads / 32; ++i) {
            if (i < w) upto += sums[i];
            total += sums[i];
        }
        int at = base + upto - __popc(used);
#pragma unroll
        for (int i = 0; i < kListEach; ++i)
            if (first + i < T) {
                const bool use = used >> i & 1;
                row[first + i] = use ? at : -1;
                if (use) src[at++] = first + i;
            }
        base += total;
        __syncthreads();
    }
    for (int i = base + threadIdx.x; i < T; i += kListThreads) src[i] = -1;
    if (threadIdx.x == 0) *count = base;
}

}  // namespace

MM_API int mm_label_rows(const long long* labels, int T, int ignore_index, int* src, int* row, int* count, cudaStream_t st) {
    label_rows_kernel<<<1, kListThreads, 0, st>>>(labels, T, ignore_index, src, row, count);
    return (int)cudaGetLastError();
}

// src, count, base: of a list of mm_label_rows whose rows from `base` on the logits belong to (labels: of all tokens), or null: row t is token t.
MM_API int mm_ce_fwd_bwd(void* logits, long long ld, const long long* labels, float* loss, int T, int V, int ignore_index, const int* src,
                         const int* count, int base, cudaStream_t st) {
    if (V % 8 || ld % 8) return -1;
    ce_fwd_bwd_kernel<<<T, kCEThreads, 0, st>>>((bf16*)logits, ld, labels, loss, V, ignore_index, src, count, base);
    return (int)cudaGetLastError();
}
