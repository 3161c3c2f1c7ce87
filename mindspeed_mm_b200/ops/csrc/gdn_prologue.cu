// Chunk-local part of the gated delta rule (WY form), forward and backward, one CTA per (chunk of 64 tokens, head), K = V = 128:
//
//   gc = cumsum(g)                                 D[i][j] = exp(gc_i - gc_j)  (j <= i)
//   A  = tril(beta_i * (k_i . k_j) * D, -1)        T = (I + A)^-1   (unit lower triangular)
//   U  = T (v * beta)          W  = T (k * beta * exp(gc))
//   Qg = q * scale * exp(gc)   Kd = k * exp(gc_last - gc)          At = (q_i . k_j) * D * scale  (j <= i)
//   gamma = exp(gc_last)
//
// Inputs are the packed [T, H, *] tensors of the layer (q, k already L2-normalised); a chunk never straddles a sequence,
// rows past the end of a sequence's last chunk are zero (beta = g = 0), so they leave T, U, W and the state untouched.
// Outputs are bf16 [H, NC, 64, *] (what the tcgen05 state-pass kernel reads) and gamma fp32 [H, NC].
//
// Arithmetic is fp32 throughout (exponentials too: this file is built without fast math), on the tensor cores where that costs
// nothing: in every 64 x 64 x 128 product one operand is a bf16 tensor as it is in memory (q, k, v, dVn, ...), and the other, if it
// is fp32 (T, dS, dP, with beta and the gates folded into its columns), is split into three bf16 terms that hold all 24 bits of it;
// products of bf16 numbers are exact in the fp32 accumulator.  (mma.sync, not tcgen05: the operands are 64 rows high and come out of
// registers and shared memory in between elementwise steps; the chain of small dependent steps, not the tensor pipe, sets the time.)
// The triangular inverse goes by 16 x 16 blocks: four diagonal blocks by substitution in registers, then three levels of block
// products with all threads, instead of 64 dependent rows.
#include "common.cuh"

namespace {

constexpr int C = 64, D = 128;
constexpr int LB = 136;                       // bf16 row stride of [64 | 128][128] tiles: ldmatrix rows fall on distinct banks
constexpr int LS = 72;                        // bf16 row stride of split [64][64] matrices
constexpr int LT = 68;                        // fp32 row stride of [64][64] matrices: rows stay 16-byte aligned
constexpr int kThreads = 256;
constexpr int kTile = C * LB * 2, kSplit = C * LS * 2, kMat = C * LT * 4;      // bytes
constexpr int kVecs = 3 * C * 4;                                              // gc, beta, exp(gc)
constexpr int kFwdSmem = 3 * kTile + 2 * kMat + kVecs + 3 * kSplit - kTile;    // the splits start in q's tile, once it is used up
constexpr int kSlots = 16;
constexpr int kBwdSmem = 7 * kTile + 2 * 2 * kTile + kVecs + kSlots * C * 4 + 64 * 4;

__device__ __forceinline__ uint32_t su32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

template <bool TRANS>
__device__ __forceinline__ void ldsm4(uint32_t* r, const bf16* p) {
    if constexpr (TRANS)
        asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
                     : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(su32(p)));
    else
        asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
                     : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(su32(p)));
}

__device__ __forceinline__ void mma16816(float* c, const uint32_t* a, uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// acc (16 rows from m0, 8 * NT columns from n0) += A B over k in [k0, k1).  A is [m][k] in memory, or [k][m] (AT); B is [n][k], or
// [k][n] (BT).  SPLITS: A is that many stacked matrices (a_step elements apart) whose sum is meant.
template <bool AT, bool BT, int NT, int SPLITS = 1>
__device__ __forceinline__ void warp_product(float (*acc)[4], const bf16* A, int lda, int m0, const bf16* B, int ldb, int n0, int k0,
                                             int k1, int a_step = 0) {
    const int lane = threadIdx.x & 31, l7 = lane & 7, b3 = (lane >> 3) & 1, b4 = lane >> 4;
    const bf16* a = AT ? A + (size_t)(l7 + b4 * 8) * lda + m0 + b3 * 8 : A + (size_t)(m0 + (lane & 15)) * lda + b4 * 8;
    const bf16* b = BT ? B + (size_t)(l7 + b3 * 8) * ldb + n0 + b4 * 8 : B + (size_t)(n0 + l7 + b4 * 8) * ldb + b3 * 8;
    for (int k = k0; k < k1; k += 16) {
        uint32_t fa[SPLITS][4];
#pragma unroll
        for (int s = 0; s < SPLITS; ++s) ldsm4<AT>(fa[s], a + s * a_step + (AT ? (size_t)k * lda : k));
#pragma unroll
        for (int n = 0; n < NT; n += 2) {
            uint32_t fb[4];
            ldsm4<BT>(fb, BT ? b + (size_t)k * ldb + n * 8 : b + (size_t)n * 8 * ldb + k);
#pragma unroll
            for (int s = 0; s < SPLITS; ++s) {
                mma16816(acc[n], fa[s], fb[0], fb[1]);
                mma16816(acc[n + 1], fa[s], fb[2], fb[3]);
            }
        }
    }
}

template <int NT>
__device__ __forceinline__ void clear(float (*acc)[4]) {
#pragma unroll
    for (int n = 0; n < NT; ++n) acc[n][0] = acc[n][1] = acc[n][2] = acc[n][3] = 0.f;
}

// x = hi + mid + lo, each a bf16 (8 + 8 + 8 bits of significand)
__device__ __forceinline__ void put_split(bf16* dst, int i, int j, float x) {
    const bf16 hi = __float2bfloat16(x);
    const float r = x - __bfloat162float(hi);
    const bf16 mid = __float2bfloat16(r);
    dst[i * LS + j] = hi;
    dst[C * LS + i * LS + j] = mid;
    dst[2 * C * LS + i * LS + j] = __float2bfloat16(r - __bfloat162float(mid));
}

// `rows` rows of 128 bf16, `pitch` elements apart in global memory -> stride LB in shared memory; rows from `len` on are zero
__device__ __forceinline__ void load_tile(bf16* dst, const bf16* src, long long pitch, int rows, int len) {
    for (int i = threadIdx.x; i < rows * 16; i += kThreads) {
        const int r = i >> 4, c = (i & 15) * 8;
        const bool in = r < len;
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(su32(dst + r * LB + c)), "l"(src + (in ? r * pitch : 0) + c),
                     "r"(in ? 16 : 0));
    }
}
__device__ __forceinline__ void loads_done() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// gc / beta / exp(gc) of the chunk (one warp scans pairs of tokens); the caller synchronises
__device__ __forceinline__ void load_gates(const float* g, const float* beta, long long tok0, int len, int H, int head, float* gc,
                                           float* bt, float* eg) {
    if (threadIdx.x >= 32) return;
    const int r = 2 * threadIdx.x;
    const float a = r < len ? g[(tok0 + r) * H + head] : 0.f, b = r + 1 < len ? g[(tok0 + r + 1) * H + head] : 0.f;
    float s = a + b;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const float t = __shfl_up_sync(0xffffffffu, s, o);
        if ((int)threadIdx.x >= o) s += t;
    }
    float before = __shfl_up_sync(0xffffffffu, s, 1);
    if (threadIdx.x == 0) before = 0.f;
    gc[r] = before + a;
    gc[r + 1] = before + a + b;
    eg[r] = expf(gc[r]);
    eg[r + 1] = expf(gc[r + 1]);
    bt[r] = r < len ? beta[(tok0 + r) * H + head] : 0.f;
    bt[r + 1] = r + 1 < len ? beta[(tok0 + r + 1) * H + head] : 0.f;
}

// T = (I + A)^-1 for the strictly lower triangular A; Y: 3 * 256 floats of scratch.  Ends synchronised.
__device__ __forceinline__ void invert(const float* A, float* T, float* Y) {
    const int t = threadIdx.x;
    if (t < C) {                                                      // diagonal blocks: a thread solves one column
        const int b = (t >> 4) * 16, c = t & 15;
        float x[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) {
            float s = i == c ? 1.f : 0.f;
#pragma unroll
            for (int j = 0; j < i; ++j) s -= A[(b + i) * LT + b + j] * x[j];       // x[j] = 0 above the column's diagonal
            x[i] = s;
        }
#pragma unroll
        for (int i = 0; i < 16; ++i) T[(b + i) * LT + b + c] = x[i];
    } else {
        for (int i = t - C; i < C * C; i += kThreads - C)
            if ((i >> 4 & 3) > (i >> 10)) T[(i >> 6) * LT + (i & 63)] = 0.f;        // blocks above the diagonal
    }
    __syncthreads();
    const int i = t >> 4, j = t & 15;
#pragma unroll
    for (int d = 1; d < 4; ++d) {
        for (int bi = d; bi < 4; ++bi) {                              // Y = sum over k of A[bi][k] T[k][bi - d]
            const int bj = bi - d;
            float s = 0.f;
#pragma unroll 16
            for (int k = bj * 16; k < bi * 16; ++k) s += A[(bi * 16 + i) * LT + k] * T[k * LT + bj * 16 + j];
            Y[(bi - d) * 256 + t] = s;
        }
        __syncthreads();
        for (int bi = d; bi < 4; ++bi) {                              // T[bi][bi - d] = -T[bi][bi] Y
            float s = 0.f;
#pragma unroll
            for (int k = 0; k < 16; ++k) s += T[(bi * 16 + i) * LT + bi * 16 + k] * Y[(bi - d) * 256 + k * 16 + j];
            T[(bi * 16 + i) * LT + (bi - d) * 16 + j] = -s;
        }
        __syncthreads();
    }
}

// 16 x 64 accumulators of a warp (rows m0 .., columns n0 ..) -> bf16 rows, `pitch` elements apart, rows below `len`
__device__ __forceinline__ void store_rows(const float (*acc)[4], bf16* dst, long long pitch, int m0, int n0, int len) {
    const int lane = threadIdx.x & 31, r = m0 + (lane >> 2), c = n0 + (lane & 3) * 2;
#pragma unroll
    for (int n = 0; n < 8; ++n) {
        if (r < len) *reinterpret_cast<bf162*>(dst + r * pitch + c + n * 8) = __floats2bfloat162_rn(acc[n][0], acc[n][1]);
        if (r + 8 < len) *reinterpret_cast<bf162*>(dst + (r + 8) * pitch + c + n * 8) = __floats2bfloat162_rn(acc[n][2], acc[n][3]);
    }
}

// Two CTAs fit an SM, so one CTA's loads and substitution run beside the other's products.  Bound by the chain of phases (load,
// scores, inverse, two products) of a CTA.  2144 chunks x heads (4096 tokens, 32 heads): 126 us; about 900 us with every product
// on CUDA cores from odd-stride fp32 tiles and a 64-row substitution by one thread per column.
__global__ void __launch_bounds__(kThreads, 2) gdn_prologue_kernel(
    const bf16* __restrict__ q, const bf16* __restrict__ k, const bf16* __restrict__ v, const float* __restrict__ g,
    const float* __restrict__ beta, const int* __restrict__ chunk_tok0, const int* __restrict__ chunk_len,
    bf16* __restrict__ W, bf16* __restrict__ Qg, bf16* __restrict__ Kd, bf16* __restrict__ At, bf16* __restrict__ U,
    float* __restrict__ gamma, int H, int NC, float scale) {
    let_successor_start();
    extern __shared__ __align__(16) uint8_t sm[];
    bf16* sK = reinterpret_cast<bf16*>(sm);
    bf16* sV = reinterpret_cast<bf16*>(sm + kTile);
    float* sA = reinterpret_cast<float*>(sm + 2 * kTile);
    float* sT = reinterpret_cast<float*>(sm + 2 * kTile + kMat);
    float* gc = reinterpret_cast<float*>(sm + 2 * kTile + 2 * kMat);
    float* bt = gc + C;
    float* eg = bt + C;
    bf16* sQ = reinterpret_cast<bf16*>(eg + C);
    bf16* sp = sQ;                                                   // splits, after q has been used
    const int c = blockIdx.x, head = blockIdx.y, len = chunk_len[c];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, m0 = (warp >> 1) * 16, wn = warp & 1;
    const long long tok0 = chunk_tok0[c], pitch = (long long)H * D, src = (tok0 * H + head) * D;
    const size_t slab = ((size_t)head * NC + c) * C;                  // row offset of this (head, chunk) in the [H, NC, 64, *] outputs
    load_tile(sK, k + src, pitch, C, len);
    load_tile(sQ, q + src, pitch, C, len);
    load_tile(sV, v + src, pitch, C, len);
    load_gates(g, beta, tok0, len, H, head, gc, bt, eg);
    loads_done();
    __syncthreads();
    if (threadIdx.x == 0) gamma[(size_t)head * NC + c] = eg[C - 1];

    {   // A and At: a warp owns 16 x 32 of both, blocks above the diagonal are only cleared
        float s[4][4], p[4][4];
        clear<4>(s);
        clear<4>(p);
        const int n0 = wn * 32;
        if (n0 <= m0 + 15) {
            warp_product<false, false, 4>(s, sK, LB, m0, sK, LB, n0, 0, D);
            warp_product<false, false, 4>(p, sQ, LB, m0, sK, LB, n0, 0, D);
        }
#pragma unroll
        for (int n = 0; n < 4; ++n)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int i = m0 + (lane >> 2) + 8 * h, j = n0 + n * 8 + (lane & 3) * 2;
                float at[2];
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    const float dec = j + e <= i ? expf(gc[i] - gc[j + e]) : 0.f;
                    sA[i * LT + j + e] = j + e < i ? bt[i] * s[n][2 * h + e] * dec : 0.f;
                    at[e] = p[n][2 * h + e] * dec * scale;
                }
                *reinterpret_cast<bf162*>(At + (slab + i) * C + j) = __floats2bfloat162_rn(at[0], at[1]);
            }
    }
    const float last = gc[C - 1];
    for (int i = threadIdx.x; i < C * (D / 8); i += kThreads) {
        const int r = i >> 4, c8 = (i & 15) * 8;
        float fq[8], fk[8];
        unpack8(*reinterpret_cast<const Vec8*>(sQ + r * LB + c8), fq);
        unpack8(*reinterpret_cast<const Vec8*>(sK + r * LB + c8), fk);
        const float a = scale * eg[r], b = expf(last - gc[r]);
#pragma unroll
        for (int e = 0; e < 8; ++e) {
            fq[e] *= a;
            fk[e] *= b;
        }
        *reinterpret_cast<Vec8*>(Qg + (slab + r) * D + c8) = pack8(fq);
        *reinterpret_cast<Vec8*>(Kd + (slab + r) * D + c8) = pack8(fk);
    }
    __syncthreads();
    invert(sA, sT, reinterpret_cast<float*>(sQ));
#pragma unroll 1
    for (int pass = 0; pass < 2; ++pass) {                            // U = (T beta) v, W = (T beta exp(gc)) k
        for (int i = threadIdx.x; i < C * C; i += kThreads) {
            const int r = i >> 6, j = i & 63;
            put_split(sp, r, j, sT[r * LT + j] * (pass ? bt[j] * eg[j] : bt[j]));
        }
        __syncthreads();
        float acc[8][4];
        clear<8>(acc);
        warp_product<false, true, 8, 3>(acc, sp, LS, m0, pass ? sK : sV, LB, wn * 64, 0, m0 + 16, C * LS);
        store_rows(acc, (pass ? W : U) + slab * D, D, m0, wn * 64, C);
        __syncthreads();
    }
}

// Sum of a row's values over the quad that holds it, left in slot[row] by one lane per row and warp column
__device__ __forceinline__ void row_slot(float a, float b, float* slot, int m0) {
#pragma unroll
    for (int o = 1; o < 4; o <<= 1) {
        a += __shfl_xor_sync(0xffffffffu, a, o);
        b += __shfl_xor_sync(0xffffffffu, b, o);
    }
    const int lane = threadIdx.x & 31, r = m0 + (lane >> 2);
    if ((lane & 3) == 0) {
        slot[r] = a;
        slot[r + 8] = b;
    }
}

// <acc row, tile row> of a warp's 16 x 64 accumulators against the same part of a bf16 tile -> slot
__device__ __forceinline__ void row_dot(const float (*acc)[4], const bf16* tile, float* slot, int m0, int n0) {
    const int lane = threadIdx.x & 31, r = m0 + (lane >> 2), c = n0 + (lane & 3) * 2;
    float a = 0.f, b = 0.f;
#pragma unroll
    for (int n = 0; n < 8; ++n) {
        const float2 x = __bfloat1622float2(*reinterpret_cast<const bf162*>(tile + r * LB + c + n * 8));
        const float2 y = __bfloat1622float2(*reinterpret_cast<const bf162*>(tile + (r + 8) * LB + c + n * 8));
        a += acc[n][0] * x.x + acc[n][1] * x.y;
        b += acc[n][2] * y.x + acc[n][3] * y.y;
    }
    row_slot(a, b, slot, m0);
}

__device__ __forceinline__ void scale_rows(float (*acc)[4], float a, float b) {
#pragma unroll
    for (int n = 0; n < 8; ++n) {
        acc[n][0] *= a;
        acc[n][1] *= a;
        acc[n][2] *= b;
        acc[n][3] *= b;
    }
}

// Backward: gradients of q, k, v, g, beta from those of the chunk's output and of the state walk.
//   dO, Vn, dVn [64, 128], Sprev^T / G^T [V, K] (state before the chunk, gradient of the state after it): bf16 [H, NC, *]
//   dW = -dVn Sprev    dQg = dO Sprev    dKd = Vn G    dAt = dO Vn^T    dU = dVn    dgamma = <G, Sprev>
//   dT = (dU v^T) beta + (dW k^T) beta exp(gc)        dA = -T^T dT T^T (strictly lower)
//   dS = dA beta_i D    dP = dAt D scale    dk = dS k + dS^T k + dP^T q + beta exp(gc) T^T dW + exp(gl - gc) dKd
//   dq = dP k + scale exp(gc) dQg           dv = beta T^T dU
// T, A and the two score matrices are recomputed; nothing of the chunk is kept in fp32 between the passes.  One CTA an SM (eleven
// 64 x 128 tiles of shared memory); bound like the forward by its chain of phases.  2144 chunks x heads: 409 us, where the batched
// products, casts, scatters and autograd through the PyTorch prologue took 4.6 ms (395 with the fast exponential).
__global__ void __launch_bounds__(kThreads, 1) gdn_prologue_bwd_kernel(
    const bf16* __restrict__ q, const bf16* __restrict__ k, const bf16* __restrict__ v, const float* __restrict__ g,
    const float* __restrict__ beta, const int* __restrict__ chunk_tok0, const int* __restrict__ chunk_len,
    const bf16* __restrict__ dO, const bf16* __restrict__ Vn, const bf16* __restrict__ dVn, const bf16* __restrict__ SprevT,
    const bf16* __restrict__ GT, bf16* __restrict__ dq, bf16* __restrict__ dk, bf16* __restrict__ dv, float* __restrict__ dg,
    float* __restrict__ dbeta, int H, int NC, float scale) {
    let_successor_start();
    extern __shared__ __align__(16) uint8_t sm[];
    auto tile = [&](int i) { return reinterpret_cast<bf16*>(sm + i * kTile); };
    bf16 *sK = tile(0), *sQ = tile(1), *sV = tile(2), *sDU = tile(3), *sDW = tile(4), *sDO = tile(5), *sVN = tile(6), *sS = tile(7), *sG = tile(9);
    float* gc = reinterpret_cast<float*>(sm + 11 * kTile);
    float* bt = gc + C;
    float* eg = bt + C;
    float* slot = eg + C;                                            // [kSlots][64]
    float* red = slot + kSlots * C;                                  // [64]
    // from the second phase on, over dO, Vn and the states: A, T (later the split of dP), dT (later dA), X, the split of T / dS
    float* sA = reinterpret_cast<float*>(sm + 5 * kTile);
    float* sT = sA + C * LT;
    float* sM = sT + C * LT;
    float* sX = sM + C * LT;
    bf16* sp = reinterpret_cast<bf16*>(sX + C * LT);
    bf16* sp2 = reinterpret_cast<bf16*>(sA);
    const int c = blockIdx.x, head = blockIdx.y, len = chunk_len[c];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, m0 = (warp >> 1) * 16, wn = warp & 1, n0 = wn * 64, h0 = wn * 32;
    const int ri = m0 + (lane >> 2);                                  // accumulator rows ri and ri + 8
    const long long tok0 = chunk_tok0[c], pitch = (long long)H * D, src = (tok0 * H + head) * D;
    const size_t slab = ((size_t)head * NC + c) * C * D, state = ((size_t)head * NC + c) * D * D;

    load_tile(sK, k + src, pitch, C, len);
    load_tile(sQ, q + src, pitch, C, len);
    load_tile(sV, v + src, pitch, C, len);
    load_tile(sDU, dVn + slab, D, C, C);
    load_tile(sDO, dO + slab, D, C, C);
    load_tile(sVN, Vn + slab, D, C, C);
    load_tile(sS, SprevT + state, D, D, D);
    load_tile(sG, GT + state, D, D, D);
    load_gates(g, beta, tok0, len, H, head, gc, bt, eg);
    loads_done();
    __syncthreads();
    const float gl = gc[C - 1], b0 = bt[ri], b1 = bt[ri + 8], e0 = eg[ri], e1 = eg[ri + 8];

    float ak[8][4], aq[8][4], dat[4][4];                              // dk, dq (16 x 64 of the warp), dAt (16 x 32)
    clear<8>(ak);
    clear<8>(aq);
    clear<4>(dat);
    warp_product<false, true, 8>(ak, sVN, LB, m0, sG, LB, n0, 0, D);
    scale_rows(ak, expf(gl - gc[ri]), expf(gl - gc[ri + 8]));
    row_dot(ak, sK, slot + (0 + wn) * C, m0, n0);                     // <dKd, Kd>
    warp_product<false, true, 8>(aq, sDO, LB, m0, sS, LB, n0, 0, D);
    scale_rows(aq, scale * e0, scale * e1);
    row_dot(aq, sQ, slot + (2 + wn) * C, m0, n0);                     // <dQg, Qg>
    if (h0 <= m0 + 15) warp_product<false, false, 4>(dat, sDO, LB, m0, sVN, LB, h0, 0, D);
    {
        float w[8][4];
        clear<8>(w);
        warp_product<false, true, 8>(w, sDU, LB, m0, sS, LB, n0, 0, D);
        scale_rows(w, -1.f, -1.f);
        store_rows(w, sDW, LB, m0, n0, C);                            // bf16, as the other operands of the walk
    }
    {
        float s = 0.f;
        for (int i = threadIdx.x; i < D * D / 8; i += kThreads) {
            float a[8], b[8];
            unpack8(*reinterpret_cast<const Vec8*>(sS + (i >> 4) * LB + (i & 15) * 8), a);
            unpack8(*reinterpret_cast<const Vec8*>(sG + (i >> 4) * LB + (i & 15) * 8), b);
#pragma unroll
            for (int e = 0; e < 8; ++e) s += a[e] * b[e];
        }
        s = warp_sum(s);
        if (lane == 0) red[warp] = s;                                 // dgamma, by warps
    }
    __syncthreads();

    // ---- scores, A, dT
    float s[4][4], p[4][4];
    clear<4>(s);
    clear<4>(p);
    if (h0 <= m0 + 15) {
        warp_product<false, false, 4>(s, sK, LB, m0, sK, LB, h0, 0, D);
        warp_product<false, false, 4>(p, sQ, LB, m0, sK, LB, h0, 0, D);
    }
#pragma unroll
    for (int n = 0; n < 4; ++n)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const int i = ri + (e >> 1) * 8, j = h0 + n * 8 + (lane & 3) * 2 + (e & 1);
            const float dec = j <= i ? expf(gc[i] - gc[j]) : 0.f;
            s[n][e] = j < i ? s[n][e] * dec : 0.f;                    // S D, strictly lower
            dat[n][e] *= dec * scale;                                 // dP, so that dAt At = dP (q_i . k_j)
            sA[i * LT + j] = s[n][e] * bt[i];
        }
    {
        float x[4][4], y[4][4];
        clear<4>(x);
        clear<4>(y);
        warp_product<false, false, 4>(x, sDU, LB, m0, sV, LB, h0, 0, D);
        warp_product<false, false, 4>(y, sDW, LB, m0, sK, LB, h0, 0, D);
#pragma unroll
        for (int n = 0; n < 4; ++n)
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const int j = h0 + n * 8 + (lane & 3) * 2 + (e & 1);
                sM[(ri + (e >> 1) * 8) * LT + j] = bt[j] * (x[n][e] + eg[j] * y[n][e]);
            }
    }
    __syncthreads();
    invert(sA, sT, sX);
    for (int i = threadIdx.x; i < C * C; i += kThreads) put_split(sp, i >> 6, i & 63, sT[(i >> 6) * LT + (i & 63)]);
    {   // X = dT T^T: rows 4 * (t / 16) .., columns t % 16 + 16 * j (rows of T, 4 banks apart); T[j][k] = 0 for k > j
        const int r0 = (threadIdx.x >> 4) * 4, cx = threadIdx.x & 15;
        float x[4][4];
        clear<4>(x);
#pragma unroll 4
        for (int kk = 0; kk < C; kk += 4) {
            float4 a[4], b[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                a[i] = *reinterpret_cast<const float4*>(sM + (r0 + i) * LT + kk);
                b[i] = *reinterpret_cast<const float4*>(sT + (cx + 16 * i) * LT + kk);
            }
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) x[i][j] += a[i].x * b[j].x + a[i].y * b[j].y + a[i].z * b[j].z + a[i].w * b[j].w;
        }
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) sX[(r0 + i) * LT + cx + 16 * j] = x[i][j];
    }
    __syncthreads();

    // ---- through T: dv, the W part of dk, dA
    {
        float w[8][4];
        clear<8>(w);
        warp_product<true, true, 8, 3>(w, sp, LS, m0, sDU, LB, n0, m0, C, C * LS);
        row_dot(w, sV, slot + (4 + wn) * C, m0, n0);
        scale_rows(w, b0, b1);
        store_rows(w, dv + src, pitch, m0, n0, len);
        clear<8>(w);
        warp_product<true, true, 8, 3>(w, sp, LS, m0, sDW, LB, n0, m0, C, C * LS);
        row_dot(w, sK, slot + (6 + wn) * C, m0, n0);
#pragma unroll
        for (int n = 0; n < 8; ++n)
#pragma unroll
            for (int e = 0; e < 4; ++e) ak[n][e] += (e < 2 ? b0 * e0 : b1 * e1) * w[n][e];
    }
    {   // dA = -T^T X, strictly lower: a 4 x 4 block a thread; T[k][i] = 0 for k < i
        const int r0 = (threadIdx.x >> 4) * 4, c0 = (threadIdx.x & 15) * 4;
        float x[4][4];
        clear<4>(x);
        if (c0 <= r0)
            for (int kk = r0; kk < C; ++kk) {
                const float4 a = *reinterpret_cast<const float4*>(sT + kk * LT + r0), b = *reinterpret_cast<const float4*>(sX + kk * LT + c0);
                const float fa[4] = {a.x, a.y, a.z, a.w}, fb[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
                for (int i = 0; i < 4; ++i)
#pragma unroll
                    for (int j = 0; j < 4; ++j) x[i][j] -= fa[i] * fb[j];
            }
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) sM[(r0 + i) * LT + c0 + j] = x[i][j];       // dT is used up
    }
    __syncthreads();

    // ---- dS, dP and the sums over rows and columns
    {
        float be0 = 0.f, be1 = 0.f, rr0 = 0.f, rr1 = 0.f;
#pragma unroll
        for (int n = 0; n < 4; ++n)
#pragma unroll
            for (int e1_ = 0; e1_ < 2; ++e1_) {
                const int j = h0 + n * 8 + (lane & 3) * 2 + e1_;
                float col = 0.f;
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const int e = 2 * h + e1_, i = ri + 8 * h;
                    const float da = j < i ? sM[i * LT + j] : 0.f, beta_i = h ? b1 : b0;
                    const float E = da * s[n][e];                     // dA S D
                    const float R = E * beta_i + dat[n][e] * p[n][e];
                    (h ? be1 : be0) += E;
                    (h ? rr1 : rr0) += R;
                    col += R;
                    put_split(sp, i, j, j < i ? da * beta_i * expf(gc[i] - gc[j]) : 0.f);
                    put_split(sp2, i, j, dat[n][e]);
                }
#pragma unroll
                for (int o = 4; o < 32; o <<= 1) col += __shfl_xor_sync(0xffffffffu, col, o);
                if (lane < 4) slot[(12 + (warp >> 1)) * C + j] = col;
            }
        row_slot(be0, be1, slot + (8 + wn) * C, m0);
        row_slot(rr0, rr1, slot + (10 + wn) * C, m0);
    }
    __syncthreads();
    warp_product<false, true, 8, 3>(ak, sp, LS, m0, sK, LB, n0, 0, m0 + 16, C * LS);          // dS k
    warp_product<true, true, 8, 3>(ak, sp, LS, m0, sK, LB, n0, m0, C, C * LS);                // dS^T k
    warp_product<true, true, 8, 3>(ak, sp2, LS, m0, sQ, LB, n0, m0, C, C * LS);               // dP^T q
    warp_product<false, true, 8, 3>(aq, sp2, LS, m0, sK, LB, n0, 0, m0 + 16, C * LS);         // dP k
    store_rows(ak, dk + src, pitch, m0, n0, len);
    store_rows(aq, dq + src, pitch, m0, n0, len);
    if (threadIdx.x < 32) {                                           // a lane has tokens 2 * lane and 2 * lane + 1
        float d[2], kd = 0.f;
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            const int i = 2 * lane + e;
            auto two = [&](int n) { return slot[n * C + i] + slot[(n + 1) * C + i]; };
            const float dkd = two(0), wk = two(6);
            kd += dkd;
            d[e] = two(2) - dkd + bt[i] * eg[i] * wk + two(10) - (two(12) + two(14));
            if (i < len) dbeta[(tok0 + i) * H + head] = two(4) + eg[i] * wk + two(8);
        }
        float dgam = 0.f;
        for (int w = 0; w < kThreads / 32; ++w) dgam += red[w];
        const float dgl = warp_sum(kd) + dgam * eg[C - 1];
        float suf = d[0] + d[1];                                      // suffix sums: g_i feeds every later gc
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const float t = __shfl_down_sync(0xffffffffu, suf, o);
            if (lane + o < 32) suf += t;
        }
        float after = __shfl_down_sync(0xffffffffu, suf, 1);
        if (lane == 31) after = 0.f;
        if (2 * lane < len) dg[(tok0 + 2 * lane) * H + head] = suf + dgl;
        if (2 * lane + 1 < len) dg[(tok0 + 2 * lane + 1) * H + head] = after + d[1] + dgl;
    }
}

// Packed [T, H, 128] <-> chunk layout [H, NC, 64, 128] (rows past a chunk's length are zero); one CTA per (chunk, head)
template <bool PACK>
__global__ void __launch_bounds__(kThreads) gdn_layout_kernel(const bf16* __restrict__ src, bf16* __restrict__ dst,
                                                              const int* __restrict__ chunk_tok0, const int* __restrict__ chunk_len, int H,
                                                              int NC) {
    let_successor_start();
    const int c = blockIdx.x, head = blockIdx.y, len = chunk_len[c];
    const size_t slab = ((size_t)head * NC + c) * C * D;
    const long long tok0 = chunk_tok0[c];
    for (int i = threadIdx.x; i < C * (D / 8); i += kThreads) {
        const int r = i >> 4, c8 = (i & 15) * 8;
        const size_t packed = ((tok0 + r) * H + head) * (size_t)D + c8, slotted = slab + r * D + c8;
        if (PACK) *reinterpret_cast<uint4*>(dst + slotted) = r < len ? *reinterpret_cast<const uint4*>(src + packed) : make_uint4(0, 0, 0, 0);
        else if (r < len) *reinterpret_cast<uint4*>(dst + packed) = *reinterpret_cast<const uint4*>(src + slotted);
    }
}

int raise_smem(const void* kern, int bytes) {
    return (int)cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
}

}  // namespace

// q, k, v: packed [T, H, 128] bf16 (heads dense, 16-byte aligned); g, beta: [T, H] fp32; chunk_tok0 / chunk_len: int32 [NC].
// W, Qg, Kd, U: bf16 [H, NC, 64, 128]; At: bf16 [H, NC, 64, 64]; gamma: fp32 [H, NC].
MM_API int mm_gdn_prologue(const void* q, const void* k, const void* v, const float* g, const float* beta,
                           const int* chunk_tok0, const int* chunk_len, void* W, void* Qg, void* Kd, void* At, void* U,
                           float* gamma, int H, int NC, float scale, cudaStream_t st) {
    if (NC == 0 || H == 0) return 0;
    if (H > 65535) return -1;
    if (int e = raise_smem((const void*)gdn_prologue_kernel, kFwdSmem)) return e;
    gdn_prologue_kernel<<<dim3(NC, H), kThreads, kFwdSmem, st>>>(
        (const bf16*)q, (const bf16*)k, (const bf16*)v, g, beta, chunk_tok0, chunk_len, (bf16*)W, (bf16*)Qg, (bf16*)Kd,
        (bf16*)At, (bf16*)U, gamma, H, NC, scale);
    return (int)cudaGetLastError();
}

// Inputs as above, dO / Vn / dVn: bf16 [H, NC, 64, 128], SprevT / GT: bf16 [H, NC, 128, 128].  dq, dk, dv: packed bf16 [T, H, 128];
// dg, dbeta: fp32 [T, H].
MM_API int mm_gdn_prologue_bwd(const void* q, const void* k, const void* v, const float* g, const float* beta, const int* chunk_tok0,
                               const int* chunk_len, const void* dO, const void* Vn, const void* dVn, const void* SprevT, const void* GT,
                               void* dq, void* dk, void* dv, float* dg, float* dbeta, int H, int NC, float scale, cudaStream_t st) {
    if (NC == 0 || H == 0) return 0;
    if (H > 65535) return -1;
    if (int e = raise_smem((const void*)gdn_prologue_bwd_kernel, kBwdSmem)) return e;
    gdn_prologue_bwd_kernel<<<dim3(NC, H), kThreads, kBwdSmem, st>>>(
        (const bf16*)q, (const bf16*)k, (const bf16*)v, g, beta, chunk_tok0, chunk_len, (const bf16*)dO, (const bf16*)Vn, (const bf16*)dVn,
        (const bf16*)SprevT, (const bf16*)GT, (bf16*)dq, (bf16*)dk, (bf16*)dv, dg, dbeta, H, NC, scale);
    return (int)cudaGetLastError();
}

// pack = 1: packed [T, H, 128] -> [H, NC, 64, 128]; pack = 0: back (rows of no chunk are left alone)
MM_API int mm_gdn_layout(const void* src, void* dst, const int* chunk_tok0, const int* chunk_len, int H, int NC, int pack, cudaStream_t st) {
    if (NC == 0 || H == 0) return 0;
    if (H > 65535) return -1;
    if (pack) gdn_layout_kernel<true><<<dim3(NC, H), kThreads, 0, st>>>((const bf16*)src, (bf16*)dst, chunk_tok0, chunk_len, H, NC);
    else gdn_layout_kernel<false><<<dim3(NC, H), kThreads, 0, st>>>((const bf16*)src, (bf16*)dst, chunk_tok0, chunk_len, H, NC);
    return (int)cudaGetLastError();
}
