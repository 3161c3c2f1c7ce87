// Generation with a key / value cache: a handful of new tokens against every weight and the whole cache.
//
// Both kernels are bound by HBM (each weight, key and value is used a few times only), and a step is a chain of some forty of
// them, most of which take 4 to 40 us, so what counts beside the bytes is how fast a kernel fills the memory system and how
// many there are.  Hence: products with M <= 4 rows stream the weights through CUDA cores instead of 128-row tensor-core tiles
// (a 128 x 256 tile grid over 3584 columns is 14 CTAs, 1.8 TB/s); the RMSNorm in front, the bias, the SwiGLU and the residual
// sum behind are part of the product; rotation, cache append and attention are one kernel.  All of them are launched with
// programmatic stream serialisation: a kernel starts while its predecessor drains, asks L2 for its first weights (a hint, so a
// predecessor that writes those weights is harmless) and waits for the predecessor before it reads anything.
#include <cooperative_groups.h>
#include <math.h>

#include "common.cuh"

namespace {

namespace cg = cooperative_groups;

__device__ __forceinline__ void prefetch_l2(const void* p) { asm volatile("prefetch.global.L2 [%0];" ::"l"(p)); }

__device__ __forceinline__ uint4 ld_once(const uint4* p) {
    uint4 v;
    asm volatile("ld.global.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
    return v;
}

__device__ __forceinline__ float2 bf2(uint32_t v) { return __bfloat1622float2(*reinterpret_cast<bf162*>(&v)); }
__device__ __forceinline__ uint32_t pack2(float a, float b) {
    bf162 t = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<uint32_t*>(&t);
}

// ------------------------------------------------------------------------------------------ skinny product
struct GemvParams {
    const bf16 *x, *w, *bias, *norm, *res;
    bf16* out;
    long long ldx, ldw, ldr, ldo;
    int N, K;                        // N: outputs (SWIGLU: half of the weight's rows)
    float eps;
};

constexpr int kGemvWarps = 4, kGemvU = 2;
constexpr int kGemvStatic = 72 * 4;                                  // static shared memory of gemv_kernel; counts towards the 48 KB

__device__ __forceinline__ void copy_async(void* smem, const void* gmem) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(smem)), "l"(gmem));
}

// out[m, n] = act(norm(x)[m, :] . w[n, :] + bias[n]) + res[m, n] for 2 to 4 rows (and one long row with a norm or SwiGLU).  A warp
// owns two weight rows (two neighbouring outputs; SWIGLU: the gate and the up row of one output), lanes stride over K in 16-byte
// pieces, the next ones of both rows in flight while the current ones are multiplied; x (normalised once per block) sits in shared
// memory as bf16, sums are fp32.  128-thread blocks: 3584 outputs are 448 blocks, so the SMs differ by one block in four.
template <int M, bool SWIGLU, bool NORM>
__global__ void __launch_bounds__(kGemvWarps * 32, M == 1 ? 8 : 4) gemv_kernel(GemvParams p) {
    extern __shared__ __align__(16) uint8_t gemv_smem[];
    bf16* xs = reinterpret_cast<bf16*>(gemv_smem);                  // [M][K]
    __shared__ float red[kGemvStatic / 4];
    const int lane = threadIdx.x & 31, nvec = p.K >> 3;
    const int unit = blockIdx.x * kGemvWarps + (threadIdx.x >> 5), units = SWIGLU ? p.N : p.N >> 1;
    const bool active = unit < units;
    const int r0 = SWIGLU ? unit : 2 * unit, r1 = SWIGLU ? p.N + unit : r0 + 1;
    const uint4* w0 = reinterpret_cast<const uint4*>(p.w + (size_t)(active ? r0 : 0) * p.ldw);
    const uint4* w1 = reinterpret_cast<const uint4*>(p.w + (size_t)(active ? r1 : 0) * p.ldw);
    if (active)
        for (int i = lane * 8; i < nvec && i < 512; i += 256) {       // 128-byte lines, the first 8 KB of each row
            prefetch_l2(w0 + i);
            prefetch_l2(w1 + i);
        }
    wait_for_predecessor();
    uint4 a[kGemvU], b[kGemvU];
    auto load = [&](int c, uint4* u, uint4* v) {
#pragma unroll
        for (int j = 0; j < kGemvU; ++j) {
            const int i = (c * kGemvU + j) * 32 + lane;
            const bool in = active && i < nvec;
            u[j] = in ? ld_once(w0 + i) : make_uint4(0, 0, 0, 0);
            v[j] = in ? ld_once(w1 + i) : make_uint4(0, 0, 0, 0);
        }
    };
    load(0, a, b);
    // every piece of x (and of the norm's weight) is in flight at once: one trip to L2, not one per loop step
    bf16* ns = xs + (size_t)M * p.K;                                 // norm weight [K]
    for (int i = threadIdx.x; i < nvec; i += kGemvWarps * 32) {
#pragma unroll
        for (int m = 0; m < M; ++m) copy_async(xs + (size_t)m * p.K + i * 8, p.x + m * p.ldx + i * 8);
        if constexpr (NORM) copy_async(ns + i * 8, p.norm + i * 8);
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    if constexpr (NORM) {
#pragma unroll
        for (int m = 0; m < M; ++m) {                                 // a thread works on the pieces that it copied
            Vec8* row = reinterpret_cast<Vec8*>(xs + (size_t)m * p.K);
            float ss = 0.f;
            for (int i = threadIdx.x; i < nvec; i += kGemvWarps * 32) {
                float f[8];
                unpack8(row[i], f);
#pragma unroll
                for (int k = 0; k < 8; ++k) ss += f[k] * f[k];
            }
            ss = block_sum(ss, red);
            const float rstd = rsqrtf(ss / (float)p.K + p.eps);
            for (int i = threadIdx.x; i < nvec; i += kGemvWarps * 32) {
                float f[8], g[8];
                unpack8(row[i], f);
                unpack8(reinterpret_cast<const Vec8*>(ns)[i], g);
#pragma unroll
                for (int k = 0; k < 8; ++k) f[k] = f[k] * rstd * g[k];
                row[i] = pack8(f);
            }
        }
    }
    __syncthreads();
    let_successor_start();
    float2 acc0[M], acc1[M];
#pragma unroll
    for (int m = 0; m < M; ++m) acc0[m] = acc1[m] = make_float2(0.f, 0.f);
    const int chunks = (nvec + 32 * kGemvU - 1) / (32 * kGemvU);
    for (int c = 0; c < chunks; ++c) {
        uint4 na[kGemvU], nb[kGemvU];
        if (c + 1 < chunks) load(c + 1, na, nb);
#pragma unroll
        for (int j = 0; j < kGemvU; ++j) {
            const int i = (c * kGemvU + j) * 32 + lane;
            const uint32_t ua[4] = {a[j].x, a[j].y, a[j].z, a[j].w}, ub[4] = {b[j].x, b[j].y, b[j].z, b[j].w};
#pragma unroll
            for (int m = 0; m < M; ++m) {
                const uint4 xv = i < nvec ? *reinterpret_cast<const uint4*>(xs + (size_t)m * p.K + i * 8) : make_uint4(0, 0, 0, 0);
                const uint32_t ux[4] = {xv.x, xv.y, xv.z, xv.w};
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    const float2 f = bf2(ux[k]);
                    acc0[m] = __ffma2_rn(bf2(ua[k]), f, acc0[m]);
                    acc1[m] = __ffma2_rn(bf2(ub[k]), f, acc1[m]);
                }
            }
        }
#pragma unroll
        for (int j = 0; j < kGemvU; ++j) {
            a[j] = na[j];
            b[j] = nb[j];
        }
    }
#pragma unroll
    for (int m = 0; m < M; ++m) {
        float s0 = warp_sum(acc0[m].x + acc0[m].y), s1 = warp_sum(acc1[m].x + acc1[m].y);
        if (lane || !active) continue;
        bf16* o = p.out + m * p.ldo;
        if constexpr (SWIGLU) {
            o[r0] = __float2bfloat16(s0 / (1.f + __expf(-s0)) * s1);
        } else {
            if (p.bias) {
                s0 += __bfloat162float(p.bias[r0]);
                s1 += __bfloat162float(p.bias[r1]);
            }
            if (p.res) {
                const float2 r = __bfloat1622float2(*reinterpret_cast<const bf162*>(p.res + m * p.ldr + r0));
                s0 += r.x;
                s1 += r.y;
            }
            *reinterpret_cast<bf162*>(o + r0) = __floats2bfloat162_rn(s0, s1);
        }
    }
}

// One row of x: the four warps of a block share pairs of weight rows (two neighbouring outputs; SWIGLU: the gate and the up row of
// one output), a quarter of K each, with the next pair (or the next piece of a long row) in flight while this one is multiplied.
// Nothing is staged: a thread's part of x stays in registers for all pairs of the block if the row is at most kRowK long, and is read
// through L1, which the weights bypass, if it is longer.  With a norm a block sums the squares of x once, while its first weights are
// on their way, and keeps the normalised x, rounded to bf16 like the norm kernel's result.
constexpr int kSplitU = 4, kStep = kGemvWarps * kSplitU * 32;        // 16-byte pieces of a row per step
constexpr int kRowK = kStep * 8;                                     // 4096
constexpr int kRowBlocks = 148 * 4;

struct RowLoads {
    uint4 a[kSplitU], b[kSplitU];
};

__device__ __forceinline__ void multiply(const RowLoads& w, const uint4* x, float2& acc0, float2& acc1) {
#pragma unroll
    for (int j = 0; j < kSplitU; ++j) {
        const uint32_t ua[4] = {w.a[j].x, w.a[j].y, w.a[j].z, w.a[j].w}, ub[4] = {w.b[j].x, w.b[j].y, w.b[j].z, w.b[j].w};
        const uint32_t ux[4] = {x[j].x, x[j].y, x[j].z, x[j].w};
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const float2 f = bf2(ux[k]);
            acc0 = __ffma2_rn(bf2(ua[k]), f, acc0);
            acc1 = __ffma2_rn(bf2(ub[k]), f, acc1);
        }
    }
}

template <bool SWIGLU>
__device__ __forceinline__ void finish_pair(const GemvParams& p, int pair, float2 s) {
    if constexpr (SWIGLU) {
        p.out[pair] = __float2bfloat16(s.x / (1.f + __expf(-s.x)) * s.y);
    } else {
        const int r = 2 * pair;
        if (p.bias) {
            s.x += __bfloat162float(p.bias[r]);
            s.y += __bfloat162float(p.bias[r + 1]);
        }
        if (p.res) {
            const float2 t = __bfloat1622float2(*reinterpret_cast<const bf162*>(p.res + r));
            s.x += t.x;
            s.y += t.y;
        }
        *reinterpret_cast<bf162*>(p.out + r) = __floats2bfloat162_rn(s.x, s.y);
    }
}

// K <= kRowK.  One wave of blocks walks the pairs.
template <bool SWIGLU, bool NORM>
__global__ void __launch_bounds__(kGemvWarps * 32, 4) gemv_rows_kernel(GemvParams p) {
    __shared__ float2 part[2][kGemvWarps];
    __shared__ float red[72];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nvec = p.K >> 3, pairs = SWIGLU ? p.N : p.N >> 1;
    auto row = [&](int pair, int second) {
        return reinterpret_cast<const uint4*>(p.w + (size_t)(SWIGLU ? pair + second * p.N : 2 * pair + second) * p.ldw);
    };
    for (int pair = blockIdx.x; pair < pairs && pair < blockIdx.x + 2 * (int)gridDim.x; pair += gridDim.x)      // the first two pairs
        for (int i = threadIdx.x * 8; i < nvec; i += kGemvWarps * 256) {
            prefetch_l2(row(pair, 0) + i);
            prefetch_l2(row(pair, 1) + i);
        }
    wait_for_predecessor();
    let_successor_start();
    auto load = [&](int pair, RowLoads& w) {
        const uint4 *w0 = row(pair, 0), *w1 = row(pair, 1);
#pragma unroll
        for (int j = 0; j < kSplitU; ++j) {
            const int i = (warp * kSplitU + j) * 32 + lane;
            w.a[j] = i < nvec ? ld_once(w0 + i) : make_uint4(0, 0, 0, 0);
            w.b[j] = i < nvec ? ld_once(w1 + i) : make_uint4(0, 0, 0, 0);
        }
    };
    RowLoads cur, nxt;
    load(blockIdx.x, cur);
    uint4 x[kSplitU];
#pragma unroll
    for (int j = 0; j < kSplitU; ++j) {
        const int i = (warp * kSplitU + j) * 32 + lane;
        x[j] = i < nvec ? reinterpret_cast<const uint4*>(p.x)[i] : make_uint4(0, 0, 0, 0);
    }
    if constexpr (NORM) {
        uint4 g[kSplitU];
        float ss = 0.f;
#pragma unroll
        for (int j = 0; j < kSplitU; ++j) {
            const int i = (warp * kSplitU + j) * 32 + lane;
            g[j] = i < nvec ? reinterpret_cast<const uint4*>(p.norm)[i] : make_uint4(0, 0, 0, 0);
            float f[8];
            unpack8(*reinterpret_cast<Vec8*>(&x[j]), f);
#pragma unroll
            for (int k = 0; k < 8; ++k) ss += f[k] * f[k];
        }
        const float rstd = rsqrtf(block_sum(ss, red) / (float)p.K + p.eps);
#pragma unroll
        for (int j = 0; j < kSplitU; ++j) {
            float f[8], h[8];
            unpack8(*reinterpret_cast<Vec8*>(&x[j]), f);
            unpack8(*reinterpret_cast<Vec8*>(&g[j]), h);
#pragma unroll
            for (int k = 0; k < 8; ++k) f[k] = f[k] * rstd * h[k];
            *reinterpret_cast<Vec8*>(&x[j]) = pack8(f);
            // past the end of the row the norm weight is zero; an infinite rstd must not turn that into NaN
            if ((warp * kSplitU + j) * 32 + lane >= nvec) x[j] = make_uint4(0, 0, 0, 0);
        }
    }
    int it = 0;
    for (int pair = blockIdx.x; pair < pairs; pair += gridDim.x, ++it) {
        if (pair + (int)gridDim.x < pairs) load(pair + gridDim.x, nxt);
        float2 acc0 = make_float2(0.f, 0.f), acc1 = make_float2(0.f, 0.f);
        multiply(cur, x, acc0, acc1);
        const float s0 = warp_sum(acc0.x + acc0.y), s1 = warp_sum(acc1.x + acc1.y);
        if (lane == 0) part[it & 1][warp] = make_float2(s0, s1);
        __syncthreads();                        // (the other half of `part` is written next: its readers are behind this barrier)
        if (threadIdx.x == (it & 3) * 32) {
            float2 s = part[it & 1][0];
#pragma unroll
            for (int w = 1; w < kGemvWarps; ++w) {
                s.x += part[it & 1][w].x;
                s.y += part[it & 1][w].y;
            }
            finish_pair<SWIGLU>(p, pair, s);
        }
        cur = nxt;
    }
}

// K > kRowK: a block per pair, the next step of both rows in flight.  3584 x 18944: 21.9 us, 6.2 TB/s (37 with a warp per pair, whose
// 12 warps an SM kept 2 KB each in flight).
__global__ void __launch_bounds__(kGemvWarps * 32) gemv_split_kernel(GemvParams p) {
    __shared__ float2 part[kGemvWarps];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nvec = p.K >> 3, pair = blockIdx.x;
    const uint4* w0 = reinterpret_cast<const uint4*>(p.w + (size_t)(2 * pair) * p.ldw);
    const uint4* w1 = reinterpret_cast<const uint4*>(p.w + (size_t)(2 * pair + 1) * p.ldw);
    const uint4* xv = reinterpret_cast<const uint4*>(p.x);
    for (int i = threadIdx.x * 8; i < nvec && i < 1024; i += kGemvWarps * 256) {       // 128-byte lines, the first 16 KB of each row
        prefetch_l2(w0 + i);
        prefetch_l2(w1 + i);
    }
    wait_for_predecessor();
    let_successor_start();
    RowLoads cur, nxt;
    uint4 x[kSplitU], nx[kSplitU];
    auto load = [&](int c, RowLoads& w, uint4* t) {
#pragma unroll
        for (int j = 0; j < kSplitU; ++j) {
            const int i = ((c * kGemvWarps + warp) * kSplitU + j) * 32 + lane;
            const bool in = i < nvec;
            w.a[j] = in ? ld_once(w0 + i) : make_uint4(0, 0, 0, 0);
            w.b[j] = in ? ld_once(w1 + i) : make_uint4(0, 0, 0, 0);
            t[j] = in ? xv[i] : make_uint4(0, 0, 0, 0);
        }
    };
    load(0, cur, x);
    float2 acc0 = make_float2(0.f, 0.f), acc1 = make_float2(0.f, 0.f);
    const int chunks = (nvec + kStep - 1) / kStep;
    for (int c = 0; c < chunks; ++c) {
        if (c + 1 < chunks) load(c + 1, nxt, nx);
        multiply(cur, x, acc0, acc1);
        cur = nxt;
#pragma unroll
        for (int j = 0; j < kSplitU; ++j) x[j] = nx[j];
    }
    const float s0 = warp_sum(acc0.x + acc0.y), s1 = warp_sum(acc1.x + acc1.y);
    if (lane == 0) part[warp] = make_float2(s0, s1);
    __syncthreads();
    if (threadIdx.x) return;
    float2 s = part[0];
#pragma unroll
    for (int w = 1; w < kGemvWarps; ++w) {
        s.x += part[w].x;
        s.y += part[w].y;
    }
    finish_pair<false>(p, pair, s);
}

template <int M, bool SWIGLU, bool NORM>
int run_gemv(const GemvParams& p, cudaStream_t st) {
    if constexpr (M == 1) {
        // one row: against a warp per pair, at the shapes of a 7B decoder layer: 4608 x 3584 with norm 12.2 -> 6.3 us, 3584 x 3584
        // 9.1 -> 5.1, 37888 x 3584 with norm and SwiGLU 48.2 -> 40.2 (6.8 TB/s), 152064 x 3584 165 -> 155, 3584 x 18944 37 -> 22
        const int pairs = SWIGLU ? p.N : p.N / 2;
        if (p.K <= kRowK)
            return launch_after(gemv_rows_kernel<SWIGLU, NORM>, 1, dim3(pairs < kRowBlocks ? pairs : kRowBlocks), kGemvWarps * 32, (size_t)0, st, p);
        if (!SWIGLU && !NORM) return launch_after(gemv_split_kernel, 1, dim3(pairs), kGemvWarps * 32, (size_t)0, st, p);
    }
    auto kern = gemv_kernel<M, SWIGLU, NORM>;
    const size_t smem = (size_t)(M + NORM) * p.K * 2;
    if (smem + kGemvStatic > 48 * 1024) {
        cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 224 * 1024);
        if (e != cudaSuccess) return (int)e;
    }
    const int units = SWIGLU ? p.N : p.N / 2;
    return launch_after(kern, 1, dim3((units + kGemvWarps - 1) / kGemvWarps), kGemvWarps * 32, smem, st, p);
}

template <int M>
int run_gemv_m(const GemvParams& p, int swiglu, cudaStream_t st) {
    if (swiglu) return p.norm ? run_gemv<M, true, true>(p, st) : run_gemv<M, true, false>(p, st);
    return p.norm ? run_gemv<M, false, true>(p, st) : run_gemv<M, false, false>(p, st);
}

// ------------------------------------------------------------------------------------------ rotary tables
// cos / sin [T, 2 * half] (both halves alike, bf16) of angle position[axis(i)][t] / theta^(i / half), axis by section.  In 64 bits: an
// angle reaches the position itself (thousands of radians), and T * half values are nothing next to the launches of the ten
// element-wise kernels that made them before, each of which a decoding step waited for.
__global__ void __launch_bounds__(128) rotary_tables_kernel(const long long* __restrict__ pos, bf16* __restrict__ cosb, bf16* __restrict__ sinb,
                                                           int T, int half, int s0, int s1, int s2, double log2_theta) {
    const int n = T * half;
    for (int j = blockIdx.x * blockDim.x + threadIdx.x; j < n; j += gridDim.x * blockDim.x) {
        const int t = j / half, i = j % half, axis = i < s0 ? 0 : i < s0 + s1 ? 1 : i < s0 + s1 + s2 ? 2 : 0;
        double s, c;
        sincos((double)pos[(size_t)axis * T + t] * exp2(-log2_theta * i / half), &s, &c);
        const bf16 cb = __float2bfloat16((float)c), sb = __float2bfloat16((float)s);
        const size_t at = (size_t)t * 2 * half + i;
        cosb[at] = cosb[at + half] = cb;
        sinb[at] = sinb[at + half] = sb;
    }
}

// ------------------------------------------------------------------------------------------ attention over the cache
struct DecodeParams {
    const bf16 *q, *k, *v;           // new tokens: [T, heads, 128] with token strides
    const bf16 *cos, *sin;           // [T, 128] or null: q and k come rotated
    const bf16 *k_old, *v_old;       // [past, Nkv, 128]
    bf16 *k_new, *v_new;             // [past + T, Nkv, 128]: cache after the call
    bf16* out;                       // [T, Nq, 128]
    long long qs, ks, vs;
    int T, past, Nq, Nkv;
    float scale_log2;
};

constexpr int kDecWarps = 8, kDecD = 128, kDecRows = 16, kDecTile = 16;
constexpr int kDecSmem = kDecWarps * kDecRows * (kDecD + 2) * 4;

__device__ __forceinline__ void mma_16x8x16(float* c, const uint32_t* a, uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// 32 consecutive elements [d0, d0 + 32) of one head of one new token, rotated (half rotation) if there are tables.
__device__ __forceinline__ void load_row32(const bf16* row, const bf16* cosr, const bf16* sinr, int d0, uint4* dst) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int d = d0 + 8 * i;
        Vec8 own = *reinterpret_cast<const Vec8*>(row + d);
        if (cosr) {
            float x[8], y[8], c[8], s[8];
            unpack8(own, x);
            unpack8(*reinterpret_cast<const Vec8*>(row + (d ^ 64)), y);
            unpack8(*reinterpret_cast<const Vec8*>(cosr + d), c);
            unpack8(*reinterpret_cast<const Vec8*>(sinr + d), s);
#pragma unroll
            for (int k = 0; k < 8; ++k) x[k] = d < 64 ? x[k] * c[k] - y[k] * s[k] : x[k] * c[k] + y[k] * s[k];
            own = pack8(x);
        }
        dst[i] = *reinterpret_cast<uint4*>(&own);
    }
}

// One cluster per key / value head, its CTAs split the keys, a warp takes every (CTAs x 8)-th run of 16 of them.  The T new tokens'
// query heads of the group (T * Nq / Nkv <= 16) are the 16 rows of an mma.sync tile: the tensor cores are used only to spare the
// cross-lane sums; the kernel moves keys and values.  Fragment order: a dot product may walk its dimension in any order, so a lane
// of a quad takes 32 consecutive elements of its key (four 16-byte loads that are also the copy into the new cache), and for the
// second product 16 consecutive elements of its four keys, paired across keys with a byte permute.  Every loaded piece is stored
// to the new cache, rotated if it belongs to a new token, so the cache is read once instead of once for the append and once for
// the attention.  Partial sums of the warps meet in shared memory, those of the CTAs in distributed shared memory: no workspace,
// no second launch.
__global__ void __launch_bounds__(kDecWarps * 32, 1) decode_attention_kernel(DecodeParams p) {
    extern __shared__ __align__(16) uint8_t dec_smem[];
    float* part_o = reinterpret_cast<float*>(dec_smem);                       // [warp][row][128]
    float* part_m = part_o + kDecWarps * kDecRows * kDecD;                    // [warp][row]
    float* part_l = part_m + kDecWarps * kDecRows;
    cg::cluster_group cluster = cg::this_cluster();
    const int splits = gridDim.x, split = blockIdx.x, kvh = blockIdx.y;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, quad = lane & 3, g = lane >> 2;
    const int G = p.Nq / p.Nkv, rows = p.T * G, L = p.past + p.T;
    const size_t pitch = (size_t)p.Nkv * kDecD;
    const int first = (split * kDecWarps + warp) * kDecTile, stride = splits * kDecWarps * kDecTile;
    for (int k0 = first; k0 < p.past; k0 += stride) {              // this warp's part of the old cache (128-byte lines) on its way to L2
        const int key = k0 + (lane >> 1);
        if (key < p.past) {
            const size_t at = key * pitch + (size_t)kvh * kDecD + (lane & 1) * 64;
            prefetch_l2(p.k_old + at);
            prefetch_l2(p.v_old + at);
        }
    }
    wait_for_predecessor();
    let_successor_start();

    // keys k0 .. k0 + 15: the lane's 32 elements of keys g and g + 8, its 16 elements of values 2 * quad (+ 1, + 8, + 9)
    auto fetch = [&](int k0, uint4 (*kk)[4], uint4 (*vv)[2]) {
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int key = k0 + h * 8 + g;
#pragma unroll
            for (int i = 0; i < 4; ++i) kk[h][i] = make_uint4(0, 0, 0, 0);
            if (key < p.past) {
                const uint4* src = reinterpret_cast<const uint4*>(p.k_old + key * pitch + (size_t)kvh * kDecD + quad * 32);
#pragma unroll
                for (int i = 0; i < 4; ++i) kk[h][i] = ld_once(src + i);
            } else if (key < L) {
                const int t = key - p.past;
                load_row32(p.k + t * p.ks + (size_t)kvh * kDecD, p.cos ? p.cos + t * kDecD : nullptr, p.sin + t * kDecD, quad * 32, kk[h]);
            }
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int key = k0 + quad * 2 + (i & 1) + (i >> 1) * 8;
            vv[i][0] = vv[i][1] = make_uint4(0, 0, 0, 0);
            if (key < L) {
                const bf16* src = key < p.past ? p.v_old + key * pitch + (size_t)kvh * kDecD : p.v + (key - p.past) * p.vs + (size_t)kvh * kDecD;
                vv[i][0] = ld_once(reinterpret_cast<const uint4*>(src + g * 16));
                vv[i][1] = ld_once(reinterpret_cast<const uint4*>(src + g * 16 + 8));
            }
        }
    };
    uint4 kk[2][4], vv[4][2];
    if (first < L) fetch(first, kk, vv);                           // in flight while the queries are read and rotated

    // query fragments: rows g and g + 8 (row = token * G + head of the group), this quad lane's 32 dims
    uint4 q0[4], q1[4];
    int vis0 = 0, vis1 = 0;                                                    // keys the two rows may see
#pragma unroll
    for (int i = 0; i < 4; ++i) q0[i] = q1[i] = make_uint4(0, 0, 0, 0);
    if (g < rows) {
        const int t = g / G;
        vis0 = p.past + t + 1;
        load_row32(p.q + t * p.qs + (size_t)(kvh * G + g % G) * kDecD, p.cos ? p.cos + t * kDecD : nullptr, p.sin + t * kDecD, quad * 32, q0);
    }
    if (g + 8 < rows) {
        const int t = (g + 8) / G;
        vis1 = p.past + t + 1;
        load_row32(p.q + t * p.qs + (size_t)(kvh * G + (g + 8) % G) * kDecD, p.cos ? p.cos + t * kDecD : nullptr, p.sin + t * kDecD, quad * 32, q1);
    }
    const uint32_t* qa = reinterpret_cast<const uint32_t*>(q0);
    const uint32_t* qb = reinterpret_cast<const uint32_t*>(q1);

    float m0 = -INFINITY, m1 = -INFINITY, l0 = 0.f, l1 = 0.f;
    float o[16][4];
#pragma unroll
    for (int n = 0; n < 16; ++n) o[n][0] = o[n][1] = o[n][2] = o[n][3] = 0.f;

    for (int k0 = first; k0 < L; k0 += stride) {
        float s[2][4];
        uint4 nk[2][4], nv[4][2];
        if (k0 + stride < L) fetch(k0 + stride, nk, nv);
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int key = k0 + h * 8 + g;
            if (key < L) {
                uint4* dst = reinterpret_cast<uint4*>(p.k_new + key * pitch + (size_t)kvh * kDecD + quad * 32);
#pragma unroll
                for (int i = 0; i < 4; ++i) dst[i] = kk[h][i];
            }
            const uint32_t* kr = reinterpret_cast<const uint32_t*>(kk[h]);
            s[h][0] = s[h][1] = s[h][2] = s[h][3] = 0.f;
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const uint32_t a[4] = {qa[2 * i], qb[2 * i], qa[2 * i + 1], qb[2 * i + 1]};
                mma_16x8x16(s[h], a, kr[2 * i], kr[2 * i + 1]);
            }
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int key = k0 + quad * 2 + (i & 1) + (i >> 1) * 8;
            if (key < L) {
                uint4* dst = reinterpret_cast<uint4*>(p.v_new + key * pitch + (size_t)kvh * kDecD + g * 16);
                dst[0] = vv[i][0];
                dst[1] = vv[i][1];
            }
        }
        float x0 = -INFINITY, x1 = -INFINITY;
#pragma unroll
        for (int h = 0; h < 2; ++h)
#pragma unroll
            for (int c = 0; c < 2; ++c) {
                const int key = k0 + h * 8 + quad * 2 + c;
                s[h][c] = key < vis0 ? s[h][c] * p.scale_log2 : -INFINITY;
                s[h][2 + c] = key < vis1 ? s[h][2 + c] * p.scale_log2 : -INFINITY;
                x0 = fmaxf(x0, s[h][c]);
                x1 = fmaxf(x1, s[h][2 + c]);
            }
#pragma unroll
        for (int d = 1; d < 4; d <<= 1) {
            x0 = fmaxf(x0, __shfl_xor_sync(0xffffffffu, x0, d));
            x1 = fmaxf(x1, __shfl_xor_sync(0xffffffffu, x1, d));
        }
        const float n0 = fmaxf(m0, x0), n1 = fmaxf(m1, x1);
        const float u0 = n0 == -INFINITY ? 0.f : n0, u1 = n1 == -INFINITY ? 0.f : n1;
        const float f0 = exp2f(m0 - u0), f1 = exp2f(m1 - u1);
        m0 = n0;
        m1 = n1;
        l0 *= f0;
        l1 *= f1;
#pragma unroll
        for (int h = 0; h < 2; ++h)
#pragma unroll
            for (int c = 0; c < 2; ++c) {
                s[h][c] = exp2f(s[h][c] - u0);
                s[h][2 + c] = exp2f(s[h][2 + c] - u1);
                l0 += s[h][c];
                l1 += s[h][2 + c];
            }
        const uint32_t pa[4] = {pack2(s[0][0], s[0][1]), pack2(s[0][2], s[0][3]), pack2(s[1][0], s[1][1]), pack2(s[1][2], s[1][3])};
        const uint32_t* v0 = reinterpret_cast<const uint32_t*>(vv[0]);
        const uint32_t* v1 = reinterpret_cast<const uint32_t*>(vv[1]);
        const uint32_t* v2 = reinterpret_cast<const uint32_t*>(vv[2]);
        const uint32_t* v3 = reinterpret_cast<const uint32_t*>(vv[3]);
#pragma unroll
        for (int n = 0; n < 16; ++n) {                                         // output column n of this lane's group: dim g * 16 + n
            const int i = n >> 1;
            const uint32_t sel = n & 1 ? 0x7632 : 0x5410;
            const uint32_t b0 = __byte_perm(v0[i], v1[i], sel), b1 = __byte_perm(v2[i], v3[i], sel);
            o[n][0] *= f0;
            o[n][1] *= f0;
            o[n][2] *= f1;
            o[n][3] *= f1;
            mma_16x8x16(o[n], pa, b0, b1);
        }
#pragma unroll
        for (int h = 0; h < 2; ++h)
#pragma unroll
            for (int i = 0; i < 4; ++i) kk[h][i] = nk[h][i];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            vv[i][0] = nv[i][0];
            vv[i][1] = nv[i][1];
        }
    }
    // Accumulator column of lane (g, quad) in product n: the output columns 2 * quad and 2 * quad + 1 of the tile, whose "column c"
    // was loaded by the lanes with group c: dims c * 16 + n.
#pragma unroll
    for (int d = 1; d < 4; d <<= 1) {
        l0 += __shfl_xor_sync(0xffffffffu, l0, d);
        l1 += __shfl_xor_sync(0xffffffffu, l1, d);
    }
    float* mo = part_o + (size_t)warp * kDecRows * kDecD;
#pragma unroll
    for (int n = 0; n < 16; ++n)
#pragma unroll
        for (int c = 0; c < 2; ++c) {
            mo[g * kDecD + (2 * quad + c) * 16 + n] = o[n][c];
            mo[(g + 8) * kDecD + (2 * quad + c) * 16 + n] = o[n][2 + c];
        }
    if (quad == 0) {
        part_m[warp * kDecRows + g] = m0;
        part_m[warp * kDecRows + g + 8] = m1;
        part_l[warp * kDecRows + g] = l0;
        part_l[warp * kDecRows + g + 8] = l1;
    }
    __syncthreads();
    // fold the warps of this CTA into warp 0's slots; the 8 factors of a row are made once, not by every element
    __shared__ float fac[16][kDecRows], all_m[kDecRows], all_l[kDecRows];      // fac: by warp here, by CTA below
    if (threadIdx.x < rows) {
        const int r = threadIdx.x;
        float m = -INFINITY, l = 0.f;
#pragma unroll
        for (int w = 0; w < kDecWarps; ++w) m = fmaxf(m, part_m[w * kDecRows + r]);
        const float u = m == -INFINITY ? 0.f : m;
#pragma unroll
        for (int w = 0; w < kDecWarps; ++w) {
            const float f = exp2f(part_m[w * kDecRows + r] - u);
            fac[w][r] = f;
            l += part_l[w * kDecRows + r] * f;
        }
        all_m[r] = m;
        all_l[r] = l;
    }
    __syncthreads();
    for (int i = threadIdx.x; i < rows * (kDecD / 4); i += kDecWarps * 32) {
        const int r = i / (kDecD / 4);
        float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int w = 0; w < kDecWarps; ++w) {
            const float4 v = reinterpret_cast<const float4*>(part_o + (size_t)w * kDecRows * kDecD)[i];
            const float f = fac[w][r];
            acc.x += v.x * f;
            acc.y += v.y * f;
            acc.z += v.z * f;
            acc.w += v.w * f;
        }
        reinterpret_cast<float4*>(part_o)[i] = acc;                            // only this thread reads or writes element i
    }
    cluster.sync();
    // fold the CTAs: each takes its share of the outputs (pairs of dims)
    if (threadIdx.x < rows) {
        const int r = threadIdx.x;
        float m = -INFINITY, l = 0.f, ms[16];
#pragma unroll
        for (int c = 0; c < 16; ++c) {
            ms[c] = c < splits ? *cluster.map_shared_rank(all_m + r, c) : -INFINITY;
            m = fmaxf(m, ms[c]);
        }
        const float u = m == -INFINITY ? 0.f : m;
#pragma unroll
        for (int c = 0; c < 16; ++c)
            if (c < splits) {
                const float f = exp2f(ms[c] - u);
                fac[c][r] = f;
                l += *cluster.map_shared_rank(all_l + r, c) * f;
            }
        part_l[r] = l > 0.f ? 1.f / l : 0.f;
    }
    __syncthreads();
    for (int i = split * kDecWarps * 32 + threadIdx.x; i < rows * (kDecD / 2); i += splits * kDecWarps * 32) {
        const int r = i / (kDecD / 2), d = i % (kDecD / 2) * 2;
        float ax = 0.f, ay = 0.f;
#pragma unroll 4
        for (int c = 0; c < splits; ++c) {
            const float2 v = *reinterpret_cast<const float2*>(cluster.map_shared_rank(part_o + r * kDecD + d, c));
            ax += v.x * fac[c][r];
            ay += v.y * fac[c][r];
        }
        const float inv = part_l[r];
        const int t = r / G, head = kvh * G + r % G;
        *reinterpret_cast<bf162*>(p.out + ((size_t)t * p.Nq + head) * kDecD + d) = __floats2bfloat162_rn(ax * inv, ay * inv);
    }
    cluster.sync();                                                            // nobody leaves while its memory is read
}

}  // namespace

// out[M, N] = swiglu?(norm?(x) @ W^T + bias?) + residual?  for M <= 4 rows.  norm: RMSNorm weight [K] or null; bias [N], res
// [M, N]: null or bf16 (not with swiglu).  swiglu: W is [2N, K], gate rows then up rows.  K % 8 == 0, N % 2 == 0, leading
// dimensions multiples of 8, 16-byte aligned bases, M * K <= 80 K elements and with a norm (M + 1) * K <= 112 K (x and the norm's
// weight in shared memory; native.skinny_supported asks for the same).
// As tensor-core tiles 3584 x 3584 and 3584 x 18944 take 25 and 83 us for one row.
MM_API int mm_gemv_bf16(const void* x, const void* w, const void* bias, const void* norm, const void* res, void* out, int M, int N,
                        int K, long long ldx, long long ldw, long long ldr, long long ldo, float eps, int swiglu, cudaStream_t st) {
    if (M < 1 || M > 4 || N < 1 || K < 1 || K % 8 || N % 2 || (ldx | ldw | ldr | ldo) % 8 || (long long)M * K > 80 * 1024 ||
        (norm && (M + 1LL) * K > 112 * 1024))
        return -1;
    if (((uintptr_t)x | (uintptr_t)w | (uintptr_t)out | (uintptr_t)norm) & 15 || ((uintptr_t)res & 3)) return -2;
    if (swiglu && (bias || res)) return -3;
    GemvParams p{(const bf16*)x, (const bf16*)w, (const bf16*)bias, (const bf16*)norm, (const bf16*)res, (bf16*)out,
                 ldx, ldw, ldr, ldo, N, K, eps};
    switch (M) {
        case 1: return run_gemv_m<1>(p, swiglu, st);
        case 2: return run_gemv_m<2>(p, swiglu, st);
        case 3: return run_gemv_m<3>(p, swiglu, st);
        default: return run_gemv_m<4>(p, swiglu, st);
    }
}

// pos: int64 [3, T]; cosb / sinb: bf16 [T, 2 * half]; sections as in the caller's model (sum <= half; what is left follows axis 0).
MM_API int mm_rotary_tables(const long long* pos, void* cosb, void* sinb, int T, int half, int s0, int s1, int s2, double theta,
                            cudaStream_t st) {
    if (T < 1 || half < 1 || (long long)T * half > 0x7fffffff || theta <= 0) return -1;
    const int blocks = (T * half + 127) / 128;
    rotary_tables_kernel<<<blocks < 148 * 8 ? blocks : 148 * 8, 128, 0, st>>>(pos, (bf16*)cosb, (bf16*)sinb, T, half, s0, s1, s2, log2(theta));
    return (int)cudaGetLastError();
}

// Appends T new tokens to a cache and attends to it (causal, aligned to the end): k_new / v_new [past + T, Nkv, 128] are the old
// cache followed by the new keys (rotated) and values.  T * Nq / Nkv <= 16; strides in elements, multiples of 8; 16-byte bases.
MM_API int mm_decode_attention(const void* q, const void* k, const void* v, const void* cos, const void* sin, const void* k_old,
                               const void* v_old, void* k_new, void* v_new, void* out, int T, int past, int Nq, int Nkv,
                               long long qs, long long ks, long long vs, float scale, cudaStream_t st) {
    if (T < 1 || past < 0 || Nkv < 1 || Nq % Nkv || (long long)T * (Nq / Nkv) > kDecRows || (qs | ks | vs) % 8 || Nkv > 65535) return -1;
    const void* ptrs[] = {q, k, v, cos, sin, k_old, v_old, k_new, v_new, out};
    for (const void* a : ptrs)
        if ((uintptr_t)a & 15) return -2;
    if (!cos != !sin) return -3;
    DecodeParams p{(const bf16*)q, (const bf16*)k, (const bf16*)v, (const bf16*)cos, (const bf16*)sin, (const bf16*)k_old,
                   (const bf16*)v_old, (bf16*)k_new, (bf16*)v_new, (bf16*)out, qs, ks, vs, T, past, Nq, Nkv,
                   scale * 1.4426950408889634f};
    // one run of 16 keys per warp before another CTA pays; 16 CTAs is the largest cluster.  More CTAs than SMs are worth it for long
    // caches only: 16 key / value heads, 16 CTAs each against 8: 2000 keys 32.4 / 28.1 us, 9000 76 / 79, 16000 111 / 132.  28 query and
    // 4 key / value heads: 311 keys 11.1 us, 2000 12.1, 9000 26.5.
    const int runs = (past + T + kDecTile * kDecWarps - 1) / (kDecTile * kDecWarps);
    int splits = 1;
    while (splits < 16 && splits < runs && (splits * 2 * Nkv <= 148 || runs >= 64)) splits *= 2;
    cudaError_t e = cudaFuncSetAttribute(decode_attention_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kDecSmem);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(decode_attention_kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    if (e != cudaSuccess) return (int)e;
    return launch_after(decode_attention_kernel, splits, dim3(splits, Nkv), kDecWarps * 32, (size_t)kDecSmem, st, p);
}
