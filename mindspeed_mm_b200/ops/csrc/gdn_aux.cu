// Auxiliary kernels of the gated-delta-net layer on packed sequences:
//   causal_conv1d (depthwise, kernel <= 8, optional SiLU, restarts at every sequence boundary) forward and backward,
//   delta_heads (the step between the convolution and the delta rule) forward and backward,
//   l2norm over the head dim (forward and backward; the gated RMSNorm of the layer's output lives in rownorm.cu).
// x is [T, D] bf16 with the channel dim contiguous and ldx elements between tokens: the convolution reads its columns of
// the fused projection in place (the seven copies of columns and heads in a training step of the layer, 4096 tokens, took
// 261 us).  A thread owns 8 channels (16 bytes) and walks a strip of tokens keeping the last K-1 inputs in registers, so
// every input is read once.
#include "common.cuh"

namespace {

constexpr int kMaxK = 8;
constexpr int kStrip = 32;   // tokens per thread strip

// seq_start[t] = first token index of the sequence token t belongs to (int32, precomputed from cu_seqlens).
// K is a template parameter so that the tap weights and the K-1 tokens of history stay in registers; the strip is
// walked in chunks of kChunk tokens whose loads are issued together.
constexpr int kChunk = 8;

template <int K, bool SILU>
__global__ void __launch_bounds__(128) conv1d_fwd_kernel(const bf16* __restrict__ x, long long ldx, const bf16* __restrict__ w,
                                                         const int* __restrict__ seq_start, bf16* __restrict__ y, int T,
                                                         int D) {
    let_successor_start();
    const int dv = D >> 3;
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= dv) return;
    const int t0 = blockIdx.y * kStrip, t1 = min(T, t0 + kStrip);
    float wk[K][8];
#pragma unroll
    for (int k = 0; k < K; ++k)
#pragma unroll
        for (int j = 0; j < 8; ++j) wk[k][j] = __bfloat162float(w[(size_t)(c * 8 + j) * K + k]);
    float hist[K][8];     // hist[i] = x[t - (K-1) + i]; hist[K-1] is the current token
    const int s0 = seq_start[t0];
#pragma unroll
    for (int i = 0; i < K - 1; ++i) {
        const int t = t0 - (K - 1) + i;
        if (t >= 0 && t >= s0) unpack8(reinterpret_cast<const Vec8*>(x + t * ldx)[c], hist[i]);
        else
#pragma unroll
            for (int j = 0; j < 8; ++j) hist[i][j] = 0.f;
    }
    for (int tc = t0; tc < t1; tc += kChunk) {
        Vec8 in[kChunk];
        int st[kChunk];
#pragma unroll
        for (int u = 0; u < kChunk; ++u)
            if (tc + u < t1) {
                in[u] = reinterpret_cast<const Vec8*>(x + (tc + u) * ldx)[c];
                st[u] = seq_start[tc + u];
            }
#pragma unroll
        for (int u = 0; u < kChunk; ++u) {
            const int t = tc + u;
            if (t >= t1) break;
            if (st[u] == t)      // a new sequence starts here: forget the history
#pragma unroll
                for (int i = 0; i < K - 1; ++i)
#pragma unroll
                    for (int j = 0; j < 8; ++j) hist[i][j] = 0.f;
            unpack8(in[u], hist[K - 1]);
            float acc[8];
#pragma unroll
            for (int j = 0; j < 8; ++j) acc[j] = 0.f;
#pragma unroll
            for (int k = 0; k < K; ++k)
#pragma unroll
                for (int j = 0; j < 8; ++j) acc[j] += wk[k][j] * hist[k][j];
            if (SILU)
#pragma unroll
                for (int j = 0; j < 8; ++j) acc[j] = acc[j] / (1.f + __expf(-acc[j]));
            reinterpret_cast<Vec8*>(y + (size_t)t * D)[c] = pack8(acc);
#pragma unroll
            for (int i = 0; i < K - 1; ++i)
#pragma unroll
                for (int j = 0; j < 8; ++j) hist[i][j] = hist[i + 1][j];
        }
    }
}

// dx[t] = sum_k w[k] * dpre[t + (K-1-k)] over outputs of the same sequence; dw[k] += dpre[u] * x[u - (K-1) + k].
// One pass over u = t0 .. t1 + K - 2 (the strip plus the K-1 outputs after it that still used its inputs): x[u] and dy[u]
// are read once, the pre-activation comes from the sliding history as in the forward, the last K values of dpre sit in a
// ring, and dx of token u - (K-1) is complete when u has been visited.  Weight gradients count outputs of the own strip
// only, so strips do not double count.
// Was bound by the latency of its loads (60% of the stalls; the registers of the windows leave 12 warps an SM), so: 4 channels a
// thread, tokens in chunks of four that are copied into shared memory three chunks ahead (each thread waits for its own copies
// only), their bounds read once a strip, and the weight gradients of the block's four strips added up in shared memory, from where
// they leave as consecutive fp32 atomics (a thread's own sums were 4.2 million, each in a 128-byte line of its own).  4096 x 8192,
// K = 4: 160 us before, 74 us now, behind a flush of L2; memory allows 29.
constexpr int kBwdWarps = 4;      // strips of a block: a warp has 128 channels of one
constexpr int kBwdChunk = 4;
constexpr int kBwdStages = 4;

__device__ __forceinline__ void copy_async8(void* smem, const void* src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"((uint32_t)__cvta_generic_to_shared(smem)), "l"(src) : "memory");
}

__device__ __forceinline__ void unpack4(const uint2& v, float* f) {
    const float2 lo = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&v.x)), hi = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&v.y));
    f[0] = lo.x, f[1] = lo.y, f[2] = hi.x, f[3] = hi.y;
}

template <int K, bool SILU>
__global__ void __launch_bounds__(32 * kBwdWarps) conv1d_bwd_kernel(const bf16* __restrict__ x, long long ldx, const bf16* __restrict__ w,
                                                                    const int* __restrict__ seq_start, const int* __restrict__ seq_end,
                                                                    const bf16* __restrict__ dy, bf16* __restrict__ dx,
                                                                    float* __restrict__ dw, int T, int D) {
    let_successor_start();
    constexpr int CH = 4;
    __shared__ uint2 stage[kBwdWarps][kBwdStages * kBwdChunk][2][32];       // x and dy of a token
    __shared__ int bounds[kBwdWarps][2][kStrip + kMaxK];                      // where the sequences of tokens t0, t0 + 1, ... start and end
    static_assert(32 * CH * kMaxK * sizeof(float) <= sizeof(stage[0]), "weight gradients lie over the stages");
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int c0 = blockIdx.x * 32 * CH, c = c0 + lane * CH;
    const int t0 = (blockIdx.y * kBwdWarps + warp) * kStrip, t1 = min(T, t0 + kStrip);
    float dwacc[K][CH];
#pragma unroll
    for (int k = 0; k < K; ++k)
#pragma unroll
        for (int j = 0; j < CH; ++j) dwacc[k][j] = 0.f;
    for (int i = lane; i < kStrip + K - 1; i += 32)
        if (t0 + i < T) {
            bounds[warp][0][i] = seq_start[t0 + i];
            bounds[warp][1][i] = min(T, seq_end[t0 + i]);
        }
    __syncwarp();
    if (c < D && t0 < T) {
        float wk[K][CH];
#pragma unroll
        for (int k = 0; k < K; ++k)
#pragma unroll
            for (int j = 0; j < CH; ++j) wk[k][j] = __bfloat162float(w[(size_t)(c + j) * K + k]);
        const bf16* xc = x + c;
        const bf16* gc = dy + c;
        const int u_end = min(T, t1 + K - 1);         // one past the last output that used an input of the strip
        uint2 (*mine)[2][32] = stage[warp];
        auto fetch = [&](int chunk) {
#pragma unroll
            for (int i = 0; i < kBwdChunk; ++i) {
                const int u = t0 + chunk * kBwdChunk + i;
                if (u < u_end) {
                    uint2 (*slot)[32] = mine[chunk % kBwdStages * kBwdChunk + i];
                    copy_async8(&slot[0][lane], xc + u * ldx);
                    copy_async8(&slot[1][lane], gc + (size_t)u * D);
                }
            }
            asm volatile("cp.async.commit_group;" ::: "memory");
        };
#pragma unroll
        for (int i = 0; i < kBwdStages - 1; ++i) fetch(i);
        float hist[K][CH];     // inputs u-(K-1) .. u (zero before the start of u's sequence)
        float ring[K][CH];     // ring[i] = dpre[u - (K-1) + i]
        const int s0 = seq_start[t0];
#pragma unroll
        for (int i = 0; i < K; ++i)
#pragma unroll
            for (int j = 0; j < CH; ++j) hist[i][j] = ring[i][j] = 0.f;
#pragma unroll
        for (int i = 0; i < K - 1; ++i) {
            const int t = t0 - (K - 1) + i;
            if (t >= 0 && t >= s0) unpack4(*reinterpret_cast<const uint2*>(xc + t * ldx), hist[i]);
        }
        for (int chunk = 0, uc = t0; uc < t1 + K - 1; ++chunk, uc += kBwdChunk) {
            fetch(chunk + kBwdStages - 1);            // (an empty group past the end) over the slots that the last chunk left
            asm volatile("cp.async.wait_group %0;" ::"n"(kBwdStages - 1) : "memory");
#pragma unroll
            for (int b = 0; b < kBwdChunk; ++b) {
                const int u = uc + b, t = u - (K - 1);
#pragma unroll
                for (int i = 0; i < K - 1; ++i)
#pragma unroll
                    for (int j = 0; j < CH; ++j) ring[i][j] = ring[i + 1][j];
                if (u < u_end) {
                    uint2 (*slot)[32] = mine[chunk % kBwdStages * kBwdChunk + b];
                    if (bounds[warp][0][u - t0] == u)
#pragma unroll
                        for (int i = 0; i < K - 1; ++i)
#pragma unroll
                            for (int j = 0; j < CH; ++j) hist[i][j] = 0.f;
                    unpack4(slot[0][lane], hist[K - 1]);
                    float g[CH];
                    unpack4(slot[1][lane], g);
                    if (SILU) {
#pragma unroll
                        for (int j = 0; j < CH; ++j) {
                            float pre = 0.f;
#pragma unroll
                            for (int k = 0; k < K; ++k) pre += wk[k][j] * hist[k][j];
                            const float sg = 1.f / (1.f + __expf(-pre));
                            g[j] = g[j] * sg * (1.f + pre * (1.f - sg));
                        }
                    }
#pragma unroll
                    for (int j = 0; j < CH; ++j) ring[K - 1][j] = g[j];
                    if (u < t1)           // weight gradient of the own strip's outputs
#pragma unroll
                        for (int k = 0; k < K; ++k)
#pragma unroll
                            for (int j = 0; j < CH; ++j) dwacc[k][j] += g[j] * hist[k][j];
#pragma unroll
                    for (int i = 0; i < K - 1; ++i)
#pragma unroll
                        for (int j = 0; j < CH; ++j) hist[i][j] = hist[i + 1][j];
                }
                // input token t has now seen all its outputs t .. t + K - 1 (ring slots 0 .. K-1), as far as its sequence goes
                if (t >= t0 && t < t1) {
                    const int e = bounds[warp][1][t - t0];
                    float acc[CH];
#pragma unroll
                    for (int j = 0; j < CH; ++j) acc[j] = 0.f;
#pragma unroll
                    for (int i = 0; i < K; ++i)            // slot i holds output t + i, which used x[t] with tap K-1-i
                        if (t + i < e)
#pragma unroll
                            for (int j = 0; j < CH; ++j) acc[j] += wk[K - 1 - i][j] * ring[i][j];
                    __nv_bfloat162 o[2] = {__floats2bfloat162_rn(acc[0], acc[1]), __floats2bfloat162_rn(acc[2], acc[3])};
                    *reinterpret_cast<uint2*>(dx + (size_t)t * D + c) = *reinterpret_cast<uint2*>(o);
                }
            }
        }
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncwarp();
    float* sdw = reinterpret_cast<float*>(stage[warp]);
#pragma unroll
    for (int j = 0; j < CH; ++j)
#pragma unroll
        for (int k = 0; k < K; ++k) sdw[(lane * CH + j) * K + k] = dwacc[k][j];
    __syncthreads();
    const int n = min(32 * CH, D - c0) * K;
    for (int i = threadIdx.x; i < n; i += 32 * kBwdWarps) {
        float sum = 0.f;
#pragma unroll
        for (int r = 0; r < kBwdWarps; ++r) sum += reinterpret_cast<const float*>(stage[r])[i];
        atomicAdd(&dw[(size_t)c0 * K + i], sum);
    }
}

// ---- l2norm over the last dim (D <= 256, one warp per row)
__global__ void l2norm_fwd_kernel(const bf16* __restrict__ x, bf16* __restrict__ y, float* __restrict__ rnorm, long long rows,
                                  int D, float eps) {
    let_successor_start();
    const long long row = (long long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (row >= rows) return;
    const int lane = threadIdx.x & 31;
    float v[8];
    float ss = 0.f;
    for (int i = lane; i < D; i += 32) {
        v[i >> 5] = __bfloat162float(x[row * D + i]);
        ss += v[i >> 5] * v[i >> 5];
    }
    ss = warp_sum(ss);
    const float r = rsqrtf(ss + eps);
    if (lane == 0 && rnorm) rnorm[row] = r;
    for (int i = lane; i < D; i += 32) y[row * D + i] = __float2bfloat16(v[i >> 5] * r);
}

__global__ void l2norm_bwd_kernel(const bf16* __restrict__ y, const bf16* __restrict__ dy, const float* __restrict__ rnorm,
                                  bf16* __restrict__ dx, long long rows, int D) {
    let_successor_start();
    const long long row = (long long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (row >= rows) return;
    const int lane = threadIdx.x & 31;
    float yv[8], gv[8];
    float dot = 0.f;
    for (int i = lane; i < D; i += 32) {
        yv[i >> 5] = __bfloat162float(y[row * D + i]);
        gv[i >> 5] = __bfloat162float(dy[row * D + i]);
        dot += yv[i >> 5] * gv[i >> 5];
    }
    dot = warp_sum(dot);
    const float r = rnorm[row];
    for (int i = lane; i < D; i += 32) dx[row * D + i] = __float2bfloat16(r * (gv[i >> 5] - yv[i >> 5] * dot));
}


// ---- the heads of the delta rule out of the convolution's result x [T, 2 hk 128 + vvec 8] = q | k | v, one CTA per token:
// q and k of hk heads L2-normalised and written rep times each (the value heads outnumber them), v copied.  Memory-bound: every byte
// is read and written once, where columns copied out, rows normalised, heads repeated and v copied out were seven passes; backward,
// the repeats' gradients are summed in fp32, go through the norm and land with dv in the one gradient of x.  T = 4096, hk = 16,
// 32 value heads: 30 us forward, where norm and copies took 160, and 35 us backward, where sums, norm and concatenation took 124.
constexpr int kHeadVec = 16;      // 16-byte vectors of a 128-wide head: half a warp per row

__device__ __forceinline__ float half_warp_sum(float v) {
#pragma unroll
    for (int o = kHeadVec / 2; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

__global__ void __launch_bounds__(256) delta_heads_fwd_kernel(const Vec8* __restrict__ x, Vec8* __restrict__ q, Vec8* __restrict__ k,
                                                              Vec8* __restrict__ v, float* __restrict__ rnorm, int hk, int rep, int vvec,
                                                              float eps) {
    let_successor_start();
    const size_t t = blockIdx.x;
    const int nn = 2 * hk * kHeadVec, W = nn + vvec;      // nn is a multiple of 32: a warp has rows to normalise or values, not both
    const Vec8* src = x + t * W;
    for (int i = threadIdx.x; i < W; i += 256) {
        Vec8 in = src[i];
        if (i >= nn) {
            v[t * vvec + (i - nn)] = in;
            continue;
        }
        float f[8];
        unpack8(in, f);
        float ss = 0.f;
#pragma unroll
        for (int j = 0; j < 8; ++j) ss += f[j] * f[j];
        const float r = rsqrtf(half_warp_sum(ss) + eps);
        const int row = i / kHeadVec, c = i % kHeadVec;
        if (c == 0) rnorm[t * 2 * hk + row] = r;
#pragma unroll
        for (int j = 0; j < 8; ++j) f[j] *= r;
        in = pack8(f);
        Vec8* dst = (row < hk ? q : k) + (t * hk + row % hk) * rep * kHeadVec + c;
        for (int j = 0; j < rep; ++j) dst[j * kHeadVec] = in;
    }
}

__global__ void __launch_bounds__(256) delta_heads_bwd_kernel(const Vec8* __restrict__ q, const Vec8* __restrict__ k,
                                                              const float* __restrict__ rnorm, const Vec8* __restrict__ dq,
                                                              const Vec8* __restrict__ dk, const Vec8* __restrict__ dv,
                                                              Vec8* __restrict__ dx, int hk, int rep, int vvec) {
    let_successor_start();
    const size_t t = blockIdx.x;
    const int nn = 2 * hk * kHeadVec, W = nn + vvec;
    Vec8* dst = dx + t * W;
    for (int i = threadIdx.x; i < W; i += 256) {
        if (i >= nn) {
            dst[i] = dv[t * vvec + (i - nn)];
            continue;
        }
        const int row = i / kHeadVec, c = i % kHeadVec;
        const size_t at = (t * hk + row % hk) * rep * kHeadVec + c;
        const Vec8* gsrc = (row < hk ? dq : dk) + at;
        float y[8], g[8];
        unpack8((row < hk ? q : k)[at], y);
        unpack8(gsrc[0], g);
        for (int j = 1; j < rep; ++j) {
            float h[8];
            unpack8(gsrc[j * kHeadVec], h);
#pragma unroll
            for (int e = 0; e < 8; ++e) g[e] += h[e];
        }
        float dot = 0.f;
#pragma unroll
        for (int e = 0; e < 8; ++e) dot += y[e] * g[e];
        dot = half_warp_sum(dot);
        const float r = rnorm[t * 2 * hk + row];
#pragma unroll
        for (int e = 0; e < 8; ++e) g[e] = r * (g[e] - y[e] * dot);
        dst[i] = pack8(g);
    }
}

}  // namespace

// x: bf16 [T, 2 hk 128 + v_width], q, k: [T, hk * rep, 128], v: [T, v_width], rnorm: fp32 [T, 2 hk]; all dense, 16-byte aligned.
MM_API int mm_delta_heads_fwd(const void* x, void* q, void* k, void* v, float* rnorm, int T, int hk, int rep, int v_width, float eps,
                              cudaStream_t st) {
    if (v_width % 8 || hk < 1 || rep < 1) return -1;
    if (T == 0) return 0;
    delta_heads_fwd_kernel<<<T, 256, 0, st>>>((const Vec8*)x, (Vec8*)q, (Vec8*)k, (Vec8*)v, rnorm, hk, rep, v_width / 8, eps);
    return (int)cudaGetLastError();
}

MM_API int mm_delta_heads_bwd(const void* q, const void* k, const float* rnorm, const void* dq, const void* dk, const void* dv, void* dx,
                              int T, int hk, int rep, int v_width, cudaStream_t st) {
    if (v_width % 8 || hk < 1 || rep < 1) return -1;
    if (T == 0) return 0;
    delta_heads_bwd_kernel<<<T, 256, 0, st>>>((const Vec8*)q, (const Vec8*)k, rnorm, (const Vec8*)dq, (const Vec8*)dk, (const Vec8*)dv,
                                              (Vec8*)dx, hk, rep, v_width / 8);
    return (int)cudaGetLastError();
}

#define MM_CONV_K(MACRO)                  \
    switch (K) {                          \
        case 1: MACRO(1); break;          \
        case 2: MACRO(2); break;          \
        case 3: MACRO(3); break;          \
        case 4: MACRO(4); break;          \
        case 5: MACRO(5); break;          \
        case 6: MACRO(6); break;          \
        case 7: MACRO(7); break;          \
        default: MACRO(8); break;         \
    }

// ldx: elements between the tokens of x, a multiple of 8.
MM_API int mm_conv1d_fwd(const void* x, long long ldx, const void* w, const int* seq_start, void* y, int T, int D, int K, int silu,
                         cudaStream_t st) {
    if (D % 8 || ldx % 8 || K > kMaxK || K < 1) return -1;
    dim3 grid((D / 8 + 127) / 128, (T + kStrip - 1) / kStrip);
#define MM_CONV_FWD(KK)                                                                                                   \
    if (silu) conv1d_fwd_kernel<KK, true><<<grid, 128, 0, st>>>((const bf16*)x, ldx, (const bf16*)w, seq_start, (bf16*)y, T, D); \
    else conv1d_fwd_kernel<KK, false><<<grid, 128, 0, st>>>((const bf16*)x, ldx, (const bf16*)w, seq_start, (bf16*)y, T, D)
    MM_CONV_K(MM_CONV_FWD)
#undef MM_CONV_FWD
    return (int)cudaGetLastError();
}

// dw: fp32 [D, K], zeroed by the caller (accumulated with atomics).
MM_API int mm_conv1d_bwd(const void* x, long long ldx, const void* w, const int* seq_start, const int* seq_end, const void* dy, void* dx,
                         float* dw, int T, int D, int K, int silu, cudaStream_t st) {
    if (D % 8 || ldx % 8 || K > kMaxK || K < 1) return -1;
    dim3 grid((D + 127) / 128, (T + kStrip * kBwdWarps - 1) / (kStrip * kBwdWarps));
#define MM_CONV_BWD(KK)                                                                                                  \
    if (silu)                                                                                                            \
        conv1d_bwd_kernel<KK, true><<<grid, 32 * kBwdWarps, 0, st>>>((const bf16*)x, ldx, (const bf16*)w, seq_start, seq_end,           \
                                                          (const bf16*)dy, (bf16*)dx, dw, T, D);                         \
    else                                                                                                                 \
        conv1d_bwd_kernel<KK, false><<<grid, 32 * kBwdWarps, 0, st>>>((const bf16*)x, ldx, (const bf16*)w, seq_start, seq_end,          \
                                                           (const bf16*)dy, (bf16*)dx, dw, T, D)
    MM_CONV_K(MM_CONV_BWD)
#undef MM_CONV_BWD
    return (int)cudaGetLastError();
}

MM_API int mm_l2norm_fwd(const void* x, void* y, float* rnorm, long long rows, int D, float eps, cudaStream_t st) {
    if (D > 256) return -1;
    l2norm_fwd_kernel<<<(unsigned)((rows + 7) / 8), 256, 0, st>>>((const bf16*)x, (bf16*)y, rnorm, rows, D, eps);
    return (int)cudaGetLastError();
}

MM_API int mm_l2norm_bwd(const void* y, const void* dy, const float* rnorm, void* dx, long long rows, int D, cudaStream_t st) {
    if (D > 256) return -1;
    l2norm_bwd_kernel<<<(unsigned)((rows + 7) / 8), 256, 0, st>>>((const bf16*)y, (const bf16*)dy, rnorm, (bf16*)dx, rows, D);
    return (int)cudaGetLastError();
}

