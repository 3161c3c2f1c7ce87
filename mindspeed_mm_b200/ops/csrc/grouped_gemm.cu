// Grouped (per-expert) bf16 GEMMs for MoE on tcgen05, all three passes, on an ALIGNED token layout:
// the rows of expert e are [off[e], off[e+1]) with every off a multiple of 128 (pad rows are zero), so no tile
// ever straddles two experts and TMA stores need no clipping.
//
//   mode 0 (fwd)   y[r, :]  = x[r, :]  @ W[e]        x [R, K]  W [E, K, N]  y [R, N]
//   mode 1 (dgrad) dx[r, :] = dy[r, :] @ W[e]^T      dy [R, N]              dx [R, K]
//   mode 2 (wgrad) dW[e]    = x_e^T @ dy_e           contraction over the expert's rows; dW [E, K, N]
//
// The persistent CTAs (TMA producer / MMA issuer / 4 epilogue warps, TMEM double buffer: same pipeline as gemm.cu; output
// tiles 128 x 256, or 128 x 128 when the tiled dimension is not a multiple of 256) number the tiles expert by expert, so
// routing skew costs nothing but the tiles it produces.  A tile's number is turned into (expert, row block, column block)
// where it is used: offsets are multiples of 128, so the row blocks before expert e are off[e] / 128 and a binary search
// over the offsets finds the expert.  (A one-thread planner kernel that wrote the list down first took 210 us a call at
// 128 experts, more than the products.)  Experts without tokens produce no rows; their wgrad tiles are written as zeros,
// so dW needs no memset before the call.  Reference op: torch_npu.npu_grouped_matmul with group_list
// (mindspeed_mm/fsdp/ops/moe_ops/gemm.py:16-92).
#include "tc05.cuh"

namespace {

using namespace tc05;

constexpr int BM = 128, BK = 64;
constexpr int kThreads = 192, kEpiThreads = 128;
constexpr int kABytes = BM * BK * 2;
constexpr int kCBytes = 2 * BM * 64 * 2;

// Output tiles are 128 x 256 when the tiled output dimension allows it (the tensor pipe reads the A tile once per 256
// columns instead of once per 128: the 128 x 128 tile is bound by shared-memory operand reads), else 128 x 128.
template <int BN>
struct Cfg {
    static constexpr int kBBytes = BN * BK * 2, kStageBytes = kABytes + kBBytes;
    static constexpr int kStages = BN == 256 ? 4 : 6;
    static constexpr int kSmem = kStages * kStageBytes + kCBytes + 2048;
    static constexpr int kTmemCols = 2 * BN;
};

struct GGParams {
    const int* off;          // [E + 1] aligned row offsets (device)
    int E, K, N;             // weight shape [E, K, N]
    int* status;
};

struct Tile {
    int e, mb, nb;           // expert, 128-row block (mode 2: block of K), column block
};

// modes 0/1: one tile per (expert row block, output column block); mode 2: per (expert, K block, N block)
template <int MODE, int BN>
__device__ __forceinline__ int tile_count(const GGParams& p) {
    if (MODE == 2) return p.E * (p.K / BM) * (p.N / BN);
    return __ldg(p.off + p.E) / BM * ((MODE == 0 ? p.N : p.K) / BN);
}

template <int MODE, int BN>
__device__ __forceinline__ Tile tile_at(const GGParams& p, int t) {
    Tile r;
    if (MODE == 2) {
        const int kb = p.K / BM, per = kb * (p.N / BN), i = t % per;
        r.e = t / per;
        r.nb = i / kb;
        r.mb = i % kb;
        return r;
    }
    const int cols = (MODE == 0 ? p.N : p.K) / BN, row = t / cols;      // row block counted over all experts
    int lo = 0, hi = p.E;                                               // off[lo] / BM <= row < off[hi] / BM
    while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (__ldg(p.off + mid) / BM <= row) lo = mid;
        else hi = mid;
    }
    const int first = __ldg(p.off + lo) / BM, rows = __ldg(p.off + hi) / BM - first, i = t - first * cols;
    r.e = lo;
    r.nb = i / rows;
    r.mb = first + i % rows;
    return r;
}

template <int MODE, int BN>
__global__ void __launch_bounds__(kThreads, 1)
grouped_gemm_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                    const __grid_constant__ CUtensorMap tmC, GGParams p) {
    constexpr int kBBytes = Cfg<BN>::kBBytes, kStageBytes = Cfg<BN>::kStageBytes, kStages = Cfg<BN>::kStages;
    constexpr int kTmemCols = Cfg<BN>::kTmemCols;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint8_t* sA = smem;
    uint8_t* sB = sA + kStages * kABytes;
    uint8_t* sC = sB + kStages * kBBytes;
    uint64_t* full = reinterpret_cast<uint64_t*>(sC + kCBytes);
    uint64_t* empty = full + kStages;
    uint64_t* tfull = empty + kStages;
    uint64_t* tempty = tfull + 2;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(tempty + 2);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
    volatile int* epi_stop = abort_flag + 1;

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int n_tiles = tile_count<MODE, BN>(p);
    auto kblocks = [&](int e) { return MODE == 2 ? (p.off[e + 1] - p.off[e]) / BK : (MODE == 0 ? p.K : p.N) / BK; };

    if (threadIdx.x == 0) {
        for (int s = 0; s < kStages; ++s) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], 1);
        }
        for (int a = 0; a < 2; ++a) {
            mbar_init(&tfull[a], 1);
            mbar_init(&tempty[a], kEpiThreads);
        }
        *abort_flag = 0;
        fence_barrier_init();
        prefetch_tmap(&tmA);
        prefetch_tmap(&tmB);
        prefetch_tmap(&tmC);
    }
    if (warp == 1) {
        tmem_alloc(tmem_slot, kTmemCols);
        tmem_relinquish();
    }
    fence_before_sync();
    __syncthreads();
    fence_after_sync();
    const uint32_t tmem_base = *tmem_slot;
    let_successor_start();           // behind the allocation, see common.cuh

    if (warp == 0) {
        if (lane == 0) {
            int stage = 0;
            uint32_t phase = 0;
            bool ok = true;
            for (int t = blockIdx.x; t < n_tiles && ok; t += gridDim.x) {
                const auto [e, mb, nb] = tile_at<MODE, BN>(p, t);
                const int kbs = kblocks(e);
                for (int kb = 0; kb < kbs; ++kb) {
                    if (!mbar_wait(&empty[stage], phase ^ 1, abort_flag)) {
                        atomicExch(p.status, MM_TIMEOUT_TMA);
                        ok = false;
                        break;
                    }
                    mbar_expect_tx(&full[stage], kStageBytes);
                    uint8_t* a = sA + stage * kABytes;
                    uint8_t* b = sB + stage * kBBytes;
                    if constexpr (MODE == 0) {
                        tma_load_2d(a, &tmA, &full[stage], kb * BK, mb * BM);
#pragma unroll
                        for (int a64 = 0; a64 < BN / 64; ++a64)                                   // W[e][k, n], N-contiguous: one
                            tma_load_3d(b + a64 * BK * 128, &tmB, &full[stage], nb * BN + 64 * a64, kb * BK, e);   // atom per 64 n
                    } else if constexpr (MODE == 1) {
                        tma_load_2d(a, &tmA, &full[stage], kb * BK, mb * BM);
                        tma_load_3d(b, &tmB, &full[stage], kb * BK, nb * BN, e);                 // rows = K (output), contraction = N
                    } else {
                        const int r0 = p.off[e] + kb * BK;
                        tma_load_2d(a, &tmA, &full[stage], mb * BM, r0);                         // x[r, k]: M = k index
                        tma_load_2d(a + BK * 128, &tmA, &full[stage], mb * BM + 64, r0);
#pragma unroll
                        for (int a64 = 0; a64 < BN / 64; ++a64)                                   // dy[r, n]
                            tma_load_2d(b + a64 * BK * 128, &tmB, &full[stage], nb * BN + 64 * a64, r0);
                    }
                    if (++stage == kStages) {
                        stage = 0;
                        phase ^= 1;
                    }
                }
            }
        }
    } else if (warp == 1) {
        if (lane == 0) {
            constexpr bool A_MN = MODE == 2, B_MN = MODE != 1;
            constexpr uint32_t idesc = idesc_bf16(BM, BN, A_MN ? 1 : 0, B_MN ? 1 : 0);
            int stage = 0, it = 0;
            uint32_t phase = 0;
            bool ok = true;
            for (int t = blockIdx.x; t < n_tiles && ok; t += gridDim.x, ++it) {
                const int kbs = kblocks(tile_at<MODE, BN>(p, t).e);
                const int acc = it & 1;
                if (!mbar_wait(&tempty[acc], ((it >> 1) & 1) ^ 1, abort_flag)) {
                    atomicExch(p.status, MM_TIMEOUT_MMA);
                    break;
                }
                fence_after_sync();
                const uint32_t d_tmem = tmem_base + acc * BN;
                for (int kb = 0; kb < kbs; ++kb) {
                    if (!mbar_wait(&full[stage], phase, abort_flag)) {
                        atomicExch(p.status, MM_TIMEOUT_MMA);
                        ok = false;
                        break;
                    }
                    fence_after_sync();
                    const uint32_t a0 = smem_u32(sA + stage * kABytes), b0 = smem_u32(sB + stage * kBBytes);
#pragma unroll
                    for (int k = 0; k < BK / 16; ++k) {
                        const uint64_t da = A_MN ? smem_desc_sw128(a0 + k * 2048, BK * 128, 1024) : smem_desc_sw128(a0 + k * 32, 16, 1024);
                        const uint64_t db = B_MN ? smem_desc_sw128(b0 + k * 2048, BK * 128, 1024) : smem_desc_sw128(b0 + k * 32, 16, 1024);
                        mma_ss(d_tmem, da, db, idesc, (kb | k) ? 1u : 0u);
                    }
                    mma_commit(&empty[stage]);
                    if (++stage == kStages) {
                        stage = 0;
                        phase ^= 1;
                    }
                }
                if (ok) mma_commit(&tfull[acc]);
            }
        }
    } else {
        const int q = warp & 3, row = q * 32 + lane;
        const bool issuer = threadIdx.x == 64;
        int it = 0, slab_count = 0;
        for (int t = blockIdx.x; t < n_tiles; t += gridDim.x, ++it) {
            const auto [e, mb, nb] = tile_at<MODE, BN>(p, t);
            const bool empty_tile = MODE == 2 && kblocks(e) == 0;       // nothing was accumulated: the tile is zero
            const int acc = it & 1;
            if (!mbar_wait(&tfull[acc], (it >> 1) & 1, abort_flag) && lane == 0) atomicExch(p.status, MM_TIMEOUT_EPI);
            asm volatile("bar.sync 1, 128;" ::: "memory");
            if (issuer) *epi_stop = *abort_flag;
            asm volatile("bar.sync 1, 128;" ::: "memory");
            if (*epi_stop) break;
            fence_after_sync();
            const uint32_t t_row = tmem_base + acc * BN + ((uint32_t)(q * 32) << 16);
#pragma unroll 1
            for (int slab = 0; slab < BN / 64; ++slab, ++slab_count) {
                uint8_t* buf = sC + (slab_count & 1) * (BM * 128);
                if (issuer) tma_wait_read<1>();
                asm volatile("bar.sync 1, 128;" ::: "memory");
                uint32_t r[64];
                tmem_ld_32x32(t_row + slab * 64, r);
                tmem_ld_32x32(t_row + slab * 64 + 32, r + 32);
                tmem_wait_ld();
                if (MODE == 2 && empty_tile) {
#pragma unroll
                    for (int j = 0; j < 64; ++j) r[j] = 0;
                }
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    uint4 v;
                    bf162 t0 = __floats2bfloat162_rn(__uint_as_float(r[8 * j + 0]), __uint_as_float(r[8 * j + 1]));
                    bf162 t1 = __floats2bfloat162_rn(__uint_as_float(r[8 * j + 2]), __uint_as_float(r[8 * j + 3]));
                    bf162 t2 = __floats2bfloat162_rn(__uint_as_float(r[8 * j + 4]), __uint_as_float(r[8 * j + 5]));
                    bf162 t3 = __floats2bfloat162_rn(__uint_as_float(r[8 * j + 6]), __uint_as_float(r[8 * j + 7]));
                    v.x = *reinterpret_cast<uint32_t*>(&t0);
                    v.y = *reinterpret_cast<uint32_t*>(&t1);
                    v.z = *reinterpret_cast<uint32_t*>(&t2);
                    v.w = *reinterpret_cast<uint32_t*>(&t3);
                    *reinterpret_cast<uint4*>(buf + row * 128 + ((j ^ (row & 7)) << 4)) = v;
                }
                fence_proxy_async();
                asm volatile("bar.sync 1, 128;" ::: "memory");
                if (issuer) {
                    if constexpr (MODE == 2) tma_store_3d(&tmC, buf, nb * BN + slab * 64, mb * BM, e);
                    else tma_store_2d(&tmC, buf, nb * BN + slab * 64, mb * BM);
                    tma_commit();
                }
            }
            fence_before_sync();
            mbar_arrive(&tempty[acc]);
        }
        if (issuer) tma_wait_all<0>();
    }

    if (*abort_flag)
        for (int i = 0; i < 64; ++i) __nanosleep(1000);
    fence_before_sync();
    __syncthreads();
    if (warp == 1) {
        fence_after_sync();
        tmem_dealloc(tmem_base, kTmemCols);
    }
}

template <int MODE, int BN>
int launch(const CUtensorMap& tA, const CUtensorMap& tB, const CUtensorMap& tC, const GGParams& p, int grid, cudaStream_t st) {
    auto kern = grouped_gemm_kernel<MODE, BN>;
    static bool done = false;
    if (!done) {
        cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg<BN>::kSmem);
        if (e != cudaSuccess) return (int)e;
        done = true;
    }
    kern<<<grid, kThreads, Cfg<BN>::kSmem, st>>>(tA, tB, tC, p);
    return (int)cudaGetLastError();
}

}  // namespace

// a, b, c by mode:  0: a = x [R,K], b = W [E,K,N], c = y [R,N]      1: a = dy [R,N], b = W, c = dx [R,K]
//                   2: a = x [R,K], b = dy [R,N], c = dW [E,K,N]
// off: int32 [E+1] on the device, multiples of 128, off[E] <= R.  K and N must be multiples of 128.  Rows from off[E] on
// are neither read nor written.
MM_API int mm_grouped_gemm_bf16(const void* a, const void* b, void* c, const int* off, int R, int E, int K, int N, int mode,
                                int* status, cudaStream_t st) {
    if (K % 128 || N % 128 || R % 128 || mode < 0 || mode > 2) return -1;
    const int BN = ((mode == 1 ? K : N) % 256 == 0) ? 256 : 128;      // the dimension the column blocks tile
    const long long max_tiles = mode == 2 ? (long long)E * (K / BM) * (N / BN) : (long long)(R / BM) * ((mode == 0 ? N : K) / BN);
    if (max_tiles > 0x7fffffffLL) return -1;
    CUtensorMap tA, tB, tC;
    int r;
    if (mode == 0) {
        if ((r = make_tmap_2d(&tA, a, R, K, K, BM, BK))) return 1000 + r;
        if ((r = make_tmap_3d(&tB, b, N, K, E, N, (uint64_t)K * N, 64, BK, 1))) return 2000 + r;
        if ((r = make_tmap_2d(&tC, c, R, N, N, BM, 64))) return 3000 + r;
    } else if (mode == 1) {
        if ((r = make_tmap_2d(&tA, a, R, N, N, BM, BK))) return 1000 + r;
        if ((r = make_tmap_3d(&tB, b, N, K, E, N, (uint64_t)K * N, BK, BN, 1))) return 2000 + r;
        if ((r = make_tmap_2d(&tC, c, R, K, K, BM, 64))) return 3000 + r;
    } else {
        if ((r = make_tmap_2d(&tA, a, R, K, K, BK, 64))) return 1000 + r;      // boxes of 64 rows (contraction) x 64 k
        if ((r = make_tmap_2d(&tB, b, R, N, N, BK, 64))) return 2000 + r;
        if ((r = make_tmap_3d(&tC, c, N, K, E, N, (uint64_t)K * N, 64, BM, 1))) return 3000 + r;
    }
    static int sms = 0;
    if (!sms) {
        int dev = 0;
        cudaGetDevice(&dev);
        if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || sms <= 0) sms = 148;
    }
    GGParams p{off, E, K, N, status};
    const int grid = max_tiles < sms ? (max_tiles < 1 ? 1 : (int)max_tiles) : sms;
    if (BN == 256) {
        if (mode == 0) return launch<0, 256>(tA, tB, tC, p, grid, st);
        if (mode == 1) return launch<1, 256>(tA, tB, tC, p, grid, st);
        return launch<2, 256>(tA, tB, tC, p, grid, st);
    }
    if (mode == 0) return launch<0, 128>(tA, tB, tC, p, grid, st);
    if (mode == 1) return launch<1, 128>(tA, tB, tC, p, grid, st);
    return launch<2, 128>(tA, tB, tC, p, grid, st);
}

// ------------------------------------------------------------------------------------------ permute / unpermute
namespace {
// dst_row[i] for every (token, slot) pair i = t * k + s, in the aligned expert-major layout; pad rows get -1 source.
__global__ void moe_permute_kernel(const bf16* __restrict__ x, const int* __restrict__ src_of_row, bf16* __restrict__ out,
                                   int R, int H) {
    let_successor_start();
    const int hv = H >> 3;
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < (long long)R * hv;
         i += (long long)gridDim.x * blockDim.x) {
        const int r = (int)(i / hv), c = (int)(i % hv);
        const int s = src_of_row[r];
        Vec8 v;
        if (s >= 0) v = reinterpret_cast<const Vec8*>(x + (size_t)s * H)[c];
        else {
#pragma unroll
            for (int k = 0; k < 4; ++k) v.v[k] = __floats2bfloat162_rn(0.f, 0.f);
        }
        reinterpret_cast<Vec8*>(out + (size_t)r * H)[c] = v;
    }
}
// out[t, :] = sum_s probs[t, s] * y[row_of_pair[t * k + s], :]   (probs null: all ones)
__global__ void moe_unpermute_kernel(const bf16* __restrict__ y, const int* __restrict__ row_of_pair,
                                     const bf16* __restrict__ probs, bf16* __restrict__ out, int T, int k, int H) {
    let_successor_start();
    const int hv = H >> 3;
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < (long long)T * hv;
         i += (long long)gridDim.x * blockDim.x) {
        const int t = (int)(i / hv), c = (int)(i % hv);
        float acc[8] = {0, 0, 0, 0, 0, 0, 0, 0};
        for (int s = 0; s < k; ++s) {
            const float w = probs ? __bfloat162float(probs[t * k + s]) : 1.f;
            float f[8];
            unpack8(reinterpret_cast<const Vec8*>(y + (size_t)row_of_pair[t * k + s] * H)[c], f);
#pragma unroll
            for (int j = 0; j < 8; ++j) acc[j] += w * f[j];
        }
        reinterpret_cast<Vec8*>(out + (size_t)t * H)[c] = pack8(acc);
    }
}

// Backward of the weighted un-permute: dy[row of (t, s)] = probs[t, s] * g[t], dprobs[t, s] = <g[t], y[row of (t, s)]>, and
// zeros in the pad rows (src_of_row < 0; null: there are none).  A warp owns a (token, slot) pair or a pad row, so every
// row of y is read once and every row of dy written once; the k warps of a token sit in one block and share its row of g in L1.
// Bound by HBM: reads y, writes dy.  4096 tokens x 8 of 2048 (49024 rows): 79 us, 4.4 TB/s; the PyTorch form
// (repeat, multiply, index_put, gather, fp32 product, sum over 0.6 GB of temporaries) took 1.1 ms.
__global__ void __launch_bounds__(256) moe_unpermute_bwd_kernel(
    const bf16* __restrict__ g, const bf16* __restrict__ y, const int* __restrict__ row_of_pair,
    const int* __restrict__ src_of_row, const bf16* __restrict__ probs, bf16* __restrict__ dy, bf16* __restrict__ dprobs,
    int pairs, int k, int R, int H) {
    let_successor_start();
    const int lane = threadIdx.x & 31, hv = H >> 3;
    const long long warps = (long long)gridDim.x * 8, total = (long long)pairs + (src_of_row ? R : 0);
    for (long long i = (long long)blockIdx.x * 8 + (threadIdx.x >> 5); i < total; i += warps) {
        if (i >= pairs) {
            const int r = (int)(i - pairs);
            if (src_of_row[r] >= 0) continue;
            uint4* dst = reinterpret_cast<uint4*>(dy + (size_t)r * H);
            for (int c = lane; c < hv; c += 32) dst[c] = make_uint4(0, 0, 0, 0);
            continue;
        }
        const Vec8* gr = reinterpret_cast<const Vec8*>(g + (size_t)(i / k) * H);
        const size_t row = (size_t)row_of_pair[i] * H;
        const Vec8* yr = reinterpret_cast<const Vec8*>(y + row);
        Vec8* dr = reinterpret_cast<Vec8*>(dy + row);
        const float w = __bfloat162float(probs[i]);
        float dot = 0.f;
#pragma unroll 4
        for (int c = lane; c < hv; c += 32) {
            float a[8], b[8];
            unpack8(gr[c], a);
            unpack8(yr[c], b);
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                dot += a[j] * b[j];
                a[j] *= w;
            }
            dr[c] = pack8(a);
        }
        dot = warp_sum(dot);
        if (lane == 0) dprobs[i] = __float2bfloat16(dot);
    }
}

// ---- routing: (token, slot) pairs -> rows of the aligned expert-major layout, pairs of an expert in their own order ----
// A counting sort: chunks of the pair list are counted by expert, the counts of an expert are summed up over the chunks, and every
// chunk places its pairs; lanes that hold the same expert find one another with match.any and warps take neighbouring pairs, so the
// order is that of a stable sort by expert.  Work is linear in pairs + experts * chunks.  With the host's
// wait for the out-of-range flag, 128 experts, 8 a token: 4096 tokens 44 us, 32768 45, 131072 63; 64, 322 and 1164 with a block per expert that
// walked the whole list, 367, 469 and 438 as radix sort, histogram and index kernels.
constexpr int kRoutePairs = 128;                 // of a warp

// hist [E][chunks]; *bad is zero beforehand.  Shared: int [E].
template <int W>
__global__ void __launch_bounds__(W * 32) moe_count_kernel(const long long* __restrict__ ids, int n, int E, int chunks, int* __restrict__ hist,
                                                           int* __restrict__ bad) {
    let_successor_start();
    extern __shared__ int route_smem[];
    for (int e = threadIdx.x; e < E; e += W * 32) route_smem[e] = 0;
    __syncthreads();
    const int first = blockIdx.x * W * kRoutePairs, last = min(n, first + W * kRoutePairs);
    for (int i = first + threadIdx.x; i < last; i += W * 32) {
        const long long e = ids[i];
        if (e < 0 || e >= E) *bad = 1;
        else atomicAdd(&route_smem[e], 1);
    }
    __syncthreads();
    for (int e = threadIdx.x; e < E; e += W * 32) hist[(size_t)e * chunks + blockIdx.x] = route_smem[e];
}

// Inclusive sum of v over the threads of a block before and including this one; `sums` holds one value per warp.  Ends synchronised.
template <int W>
__device__ __forceinline__ int block_scan(int v, int* sums, int& total) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int t = __shfl_up_sync(0xffffffffu, v, o);
        if (lane >= o) v += t;
    }
    if (lane == 31) sums[w] = v;
    __syncthreads();
    total = 0;
#pragma unroll
    for (int i = 0; i < W; ++i) {
        if (i < w) v += sums[i];
        total += sums[i];
    }
    __syncthreads();
    return v;
}

// One block per expert: counts by chunk -> pairs in the chunks before; counts[e]: all of them
__global__ void __launch_bounds__(256) moe_scan_kernel(int* __restrict__ hist, int chunks, int* __restrict__ counts) {
    let_successor_start();
    __shared__ int sums[8];
    int* h = hist + (size_t)blockIdx.x * chunks;
    int base = 0;
    for (int c0 = 0; c0 < chunks; c0 += 256) {
        const int c = c0 + threadIdx.x, v = c < chunks ? h[c] : 0;
        int total;
        const int upto = block_scan<8>(v, sums, total);
        if (c < chunks) h[c] = base + upto - v;
        base += total;
    }
    if (threadIdx.x == 0) counts[blockIdx.x] = base;
}

// hist: pairs of the expert in the chunks before, or null for a single chunk.  Shared: int [W][E].
template <int W>
__global__ void __launch_bounds__(W * 32) moe_place_kernel(const long long* __restrict__ ids, int n, int k, int E, int chunks,
                                                           const int* __restrict__ hist, const int* __restrict__ counts, int R,
                                                           int* __restrict__ off, int* __restrict__ row_of_pair, int* __restrict__ src_of_row) {
    let_successor_start();
    extern __shared__ int route_smem[];
    __shared__ int sums[W];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    int* mine = route_smem + (size_t)w * E;               // this warp's pairs of each expert, then where the next one goes
    for (int i = threadIdx.x; i < W * E; i += W * 32) route_smem[i] = 0;
    __syncthreads();
    const int first = (blockIdx.x * W + w) * kRoutePairs;
    int key[kRoutePairs / 32];
    unsigned peers[kRoutePairs / 32];
#pragma unroll
    for (int j = 0; j < kRoutePairs / 32; ++j) {
        const int i = first + j * 32 + lane;
        const long long e = i < n ? ids[i] : -1;
        key[j] = e >= 0 && e < E ? (int)e : -1;
        peers[j] = __match_any_sync(0xffffffffu, key[j]);
        if (key[j] >= 0 && lane == __ffs(peers[j]) - 1) mine[key[j]] += __popc(peers[j]);
        __syncwarp();
    }
    __syncthreads();
    int start = 0;                                        // first row of the experts of this step
    for (int e0 = 0; e0 < E; e0 += W * 32) {
        const int e = e0 + threadIdx.x, count = e < E ? counts[e] : 0, padded = (count + 127) / 128 * 128;
        int total;
        const int at = start + block_scan<W>(padded, sums, total) - padded;
        if (e < E) {
            int run = at + (hist ? hist[(size_t)e * chunks + blockIdx.x] : 0);
            for (int i = 0; i < W; ++i) {
                const int c = route_smem[(size_t)i * E + e];
                route_smem[(size_t)i * E + e] = run;
                run += c;
            }
            if (blockIdx.x == 0) off[e] = at;
            if (e % gridDim.x == blockIdx.x)
                for (int r = at + count; r < at + padded; ++r) src_of_row[r] = -1;
        }
        start += total;
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) off[E] = start;
    for (int r = start + blockIdx.x * W * 32 + threadIdx.x; r < R; r += gridDim.x * W * 32) src_of_row[r] = -1;      // rows that no expert uses
    __syncthreads();
#pragma unroll
    for (int j = 0; j < kRoutePairs / 32; ++j) {
        const int i = first + j * 32 + lane;
        const int r = key[j] >= 0 ? mine[key[j]] + __popc(peers[j] & ((1u << lane) - 1)) : 0;
        __syncwarp();
        if (key[j] >= 0) {
            if (lane == __ffs(peers[j]) - 1) mine[key[j]] += __popc(peers[j]);
            row_of_pair[i] = r;
            src_of_row[r] = i / k;
        }
        __syncwarp();
    }
}

// Eight warps a block, or one where the experts' places of eight do not fit shared memory.
inline int route_warps(int E) { return E <= 6000 ? 8 : 1; }
inline int route_chunks(int n, int E) {
    const int pairs = route_warps(E) * kRoutePairs;
    return n > 0 ? (n - 1) / pairs + 1 : 1;
}

template <int W>
int route(const long long* ids, int n, int k, int E, int R, int* scratch, int* off, int* row_of_pair, int* src_of_row, int* bad, cudaStream_t st) {
    const int chunks = route_chunks(n, E), smem = E * 4;
    int *counts = scratch, *hist = scratch + E;
    if (smem > 48 * 1024) {
        const cudaError_t e = cudaFuncSetAttribute(moe_count_kernel<W>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
        if (e != cudaSuccess) return (int)e;
    }
    if (W * smem + W * 4 > 48 * 1024) {
        const cudaError_t e = cudaFuncSetAttribute(moe_place_kernel<W>, cudaFuncAttributeMaxDynamicSharedMemorySize, W * smem);
        if (e != cudaSuccess) return (int)e;
    }
    if (chunks == 1) {                                    // the counts of the one chunk are the experts' own
        moe_count_kernel<W><<<1, W * 32, smem, st>>>(ids, n, E, 1, counts, bad);
        hist = nullptr;
    } else {
        moe_count_kernel<W><<<chunks, W * 32, smem, st>>>(ids, n, E, chunks, hist, bad);
        moe_scan_kernel<<<E, 256, 0, st>>>(hist, chunks, counts);
    }
    moe_place_kernel<W><<<chunks, W * 32, W * smem, st>>>(ids, n, k, E, chunks, hist, counts, R, off, row_of_pair, src_of_row);
    return (int)cudaGetLastError();
}
}  // namespace

MM_API int mm_moe_permute(const void* x, const int* src_of_row, void* out, int R, int H, cudaStream_t st) {
    if (H % 8) return -1;
    long long work = (long long)R * (H / 8);
    int grid = (int)((work + 255) / 256 < 148 * 16 ? (work + 255) / 256 : 148 * 16);
    moe_permute_kernel<<<grid < 1 ? 1 : grid, 256, 0, st>>>((const bf16*)x, src_of_row, (bf16*)out, R, H);
    return (int)cudaGetLastError();
}

MM_API int mm_moe_unpermute(const void* y, const int* row_of_pair, const void* probs, void* out, int T, int k, int H,
                            cudaStream_t st) {
    if (H % 8) return -1;
    long long work = (long long)T * (H / 8);
    int grid = (int)((work + 255) / 256 < 148 * 16 ? (work + 255) / 256 : 148 * 16);
    moe_unpermute_kernel<<<grid < 1 ? 1 : grid, 256, 0, st>>>((const bf16*)y, row_of_pair, (const bf16*)probs, (bf16*)out, T, k, H);
    return (int)cudaGetLastError();
}

MM_API int mm_moe_unpermute_bwd(const void* g, const void* y, const int* row_of_pair, const int* src_of_row, const void* probs,
                                void* dy, void* dprobs, int T, int k, int R, int H, cudaStream_t st) {
    if (H % 8) return -1;
    if (!T && !src_of_row) return 0;
    const long long warps = (long long)T * k + (src_of_row ? R : 0), blocks = (warps + 7) / 8;
    const int grid = (int)(blocks < 148 * 8 ? (blocks < 1 ? 1 : blocks) : 148 * 8);
    moe_unpermute_bwd_kernel<<<grid, 256, 0, st>>>((const bf16*)g, (const bf16*)y, row_of_pair, src_of_row, (const bf16*)probs,
                                                  (bf16*)dy, (bf16*)dprobs, T * k, k, R, H);
    return (int)cudaGetLastError();
}

// Ints of scratch for mm_moe_route.
MM_API long long mm_moe_route_scratch(int n, int E) { return E < 1 ? 0 : E + (long long)E * route_chunks(n, E); }

// ids: n = T * k expert numbers.  Writes off [E + 1], row_of_pair [n], src_of_row [R] (-1: pad row) with
// R >= n + 127 * E, and *bad = 1 when an id lies outside [0, E).  The caller zeroes *bad, and row_of_pair, in which such a pair is
// not written.
MM_API int mm_moe_route(const long long* ids, int n, int k, int E, int R, int* scratch, int* off, int* row_of_pair,
                        int* src_of_row, int* bad, cudaStream_t st) {
    if (E < 1 || E > 56000 || k < 1 || R < n) return -1;
    return route_warps(E) == 8 ? route<8>(ids, n, k, E, R, scratch, off, row_of_pair, src_of_row, bad, st)
                               : route<1>(ids, n, k, E, R, scratch, off, row_of_pair, src_of_row, bad, st);
}
