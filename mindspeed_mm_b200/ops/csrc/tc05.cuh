// Inline-PTX wrappers for the Blackwell (sm_100a) data path: mbarrier, TMA (cp.async.bulk.tensor),
// tcgen05 MMA / TMEM alloc / TMEM load, and the UMMA shared-memory / instruction descriptors.
//
// Every wait in here is BOUNDED: a wait that runs out returns false, the caller records a status word
// and unwinds (frees TMEM, returns).  Nothing traps and nothing spins forever.
#pragma once
#include <cuda.h>
#include "common.cuh"

namespace tc05 {

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ bool elect_one() {
    uint32_t pred = 0;
    asm volatile(
        "{\n"
        ".reg .b32 %%rx;\n"
        ".reg .pred %%px;\n"
        "elect.sync %%rx|%%px, %1;\n"
        "@%%px mov.s32 %0, 1;\n"
        "}\n"
        : "+r"(pred)
        : "r"(0xffffffffu));
    return pred != 0;
}

// ------------------------------------------------------------------------------------------ mbarrier
__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count));
}
__device__ __forceinline__ void fence_barrier_init() { asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory"); }
__device__ __forceinline__ void fence_proxy_async() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n"
        ".reg .pred p;\n"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
        "selp.u32 %0, 1, 0, p;\n"
        "}\n"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}

// Bounded wait.  `abort_flag` (shared) lets one timed-out role release the others at once.
// ~2^31 cycles (about one second at 1.9 GHz) before giving up.
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity, volatile int* abort_flag) {
    if (mbar_try_wait(bar, parity)) return true;
    const long long t0 = clock64();
    while (true) {
        for (int i = 0; i < 64; ++i)
            if (mbar_try_wait(bar, parity)) return true;
        if (*abort_flag) return false;
        if (clock64() - t0 > (1LL << 31)) {
            *abort_flag = 1;
            return false;
        }
    }
}

// ------------------------------------------------------------------------------------------ pairs of CTAs
// Two CTAs of a cluster work on one tile (cta_group::2).  Barriers that both write live in the CTA of rank 0.
__device__ __forceinline__ uint32_t cluster_rank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
// address of the same shared-memory variable in CTA `rank` of the cluster
__device__ __forceinline__ uint32_t cluster_addr(const void* p, uint32_t rank) {
    uint32_t a;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(smem_u32(p)), "r"(rank));
    return a;
}
__device__ __forceinline__ void cluster_sync() {
    asm volatile("barrier.cluster.arrive.release;\nbarrier.cluster.wait.acquire;" ::: "memory");
}
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t bar) {
    asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait_cluster(uint64_t* bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n"
        ".reg .pred p;\n"
        "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n"
        "selp.u32 %0, 1, 0, p;\n"
        "}\n"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}
// mbar_wait for a barrier that threads of the other CTA arrive on
__device__ __forceinline__ bool mbar_wait_cluster(uint64_t* bar, uint32_t parity, volatile int* abort_flag) {
    const long long t0 = clock64();
    while (true) {
        for (int i = 0; i < 64; ++i)
            if (mbar_try_wait_cluster(bar, parity)) return true;
        if (*abort_flag) return false;
        if (clock64() - t0 > (1LL << 31)) {
            *abort_flag = 1;
            return false;
        }
    }
}

// ------------------------------------------------------------------------------------------ packed attention tiles
// Non-causal self-attention over many short sequences (vision-tower windows of 64 tokens): a tile may cover several
// whole consecutive sequences whose lengths add up to at most its 128 rows.  The kernels then treat the group as one
// sequence and mask block-diagonally: a row that belongs to sequence s only sees [cu[s], cu[s+1]).  `tok` is the row's
// packed token index, `begin` = cu[first]; the range comes back relative to `begin`.
__device__ __forceinline__ void packed_row_range(const int* cu, int first, int nseq, int tok, int begin, int& lo, int& hi) {
    for (int s = first; s < first + nseq; ++s) {
        const int a = cu[s], b = cu[s + 1];
        if (tok >= a && tok < b) {
            lo = a - begin;
            hi = b - begin;
        }
    }
}

// Attention tile list of one kernel, written by one block.
//   pack: sequences in their order; one of at least `rows` rows is cut into tiles, a shorter one shares its tile with as many
//         following ones as fit (the greedy walk is serial in the tiles; all threads look for the ends).
//   else: tiles of all sequences by their position t in the sequence, `descending` from the last one (causal attention: the tiles
//         with most work first).  Position by position, the block keeps the sequences that reach it and ranks them by ballot, which is
//         linear in the tiles; once kPlanFew sequences or fewer are left, their tiles find their places independently of one another.
// Offsets that reach past the tensors make more tiles than the list holds; none is listed then.
// Forward / backward in us, causal, 2 heads of 64: one thread with the offsets in global memory; every tile counting the tiles of all
// sequences; this.  4 x 2048: 42 / 148, 37 / 126, 37 / 121.  512 x 16: 85 / 181, 697 / 1769, 59 / 112.  4096 x 2: 608 / 1273,
// 41030 / 105651, 321 / 642.  128 windows of 64 without a mask: 42 / 113 with one thread, 31 / 100 now.
constexpr int kPlanThreads = 256, kPlanWarps = kPlanThreads / 32, kPlanCache = 4096, kPlanFew = 32;
__device__ __forceinline__ void plan_tiles(const int* cu, int n_seqs, int* tile_seq, int* tile_r0, int* n_tiles, int* tile_nseq,
                                           int max_tiles, int rows, bool descending, bool pack) {
    __shared__ int cached[kPlanCache + 1], list[kPlanCache];
    const bool fits = n_seqs <= kPlanCache;
    if (fits)
        for (int i = threadIdx.x; i <= n_seqs; i += kPlanThreads) cached[i] = cu[i];
    __syncthreads();
    const int* off = fits ? cached : cu;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (pack) {
        // where a tile that starts at sequence b ends, for every b; the walk from end to end is then a read per tile
        auto end_of = [&](int b) {
            int e = b + 1;
            while (e < n_seqs && off[e + 1] - off[b] <= rows) ++e;
            return e;
        };
        if (fits)
            for (int b = threadIdx.x; b < n_seqs; b += kPlanThreads) list[b] = end_of(b);
        __syncthreads();
        if (warp) return;
        int n = 0;
        for (int b = 0; b < n_seqs && n < max_tiles;) {
            const int len = off[b + 1] - off[b], end = fits ? list[b] : end_of(b);
            if (len >= rows) {
                const int cut = min((len + rows - 1) / rows, max_tiles - n);
                for (int t = lane; t < cut; t += 32) {
                    tile_seq[n + t] = b;
                    tile_r0[n + t] = t * rows;
                    tile_nseq[n + t] = 1;
                }
                n += cut;
                ++b;
                continue;
            }
            if (lane == 0) {
                tile_seq[n] = b;
                tile_r0[n] = 0;
                tile_nseq[n] = end - b;
            }
            ++n;
            b = end;
        }
        if (lane == 0) *n_tiles = n;
        return;
    }
    __shared__ int warp_count[kPlanWarps], few_seq[kPlanFew], few_tiles[kPlanFew];
    __shared__ unsigned long long sum;
    auto tiles = [&](int b) { return max(0, (off[b + 1] - off[b] + rows - 1) / rows); };
    if (threadIdx.x == 0) sum = 0;
    __syncthreads();
    unsigned long long mine = 0;
    for (int b = threadIdx.x; b < n_seqs; b += kPlanThreads) mine += tiles(b);
    if (mine) atomicAdd(&sum, mine);
    __syncthreads();
    const int total = sum <= (unsigned long long)max_tiles ? (int)sum : 0;
    if (threadIdx.x == 0) *n_tiles = total;
    if (!total) return;
    auto place = [&](int k) { return descending ? total - 1 - k : k; };      // of the k-th tile by rising position
    auto put = [&](int k, int b, int t) {
        const int at = place(k);
        tile_seq[at] = b;
        tile_r0[at] = t * rows;
        tile_nseq[at] = 1;
    };
    // count: sequences with more than t - 1 tiles, in `list` or, where that is too short, in the tile list at position t - 1
    int t = 0, count = n_seqs, k0 = 0, before_k0 = 0;
    auto candidate = [&](int i) { return t == 0 ? i : fits ? list[i] : tile_seq[place(before_k0 + i)]; };
    while (count > kPlanFew) {
        int kept = 0;
        for (int i0 = 0; i0 < count; i0 += kPlanThreads) {
            const int i = i0 + threadIdx.x, b = i < count ? candidate(i) : 0;
            const bool keep = i < count && tiles(b) > t;
            const unsigned m = __ballot_sync(0xffffffffu, keep);
            if (lane == 0) warp_count[warp] = __popc(m);
            __syncthreads();                         // the candidates of this stretch are read, too: `list` is compacted in place
            int rank = kept + __popc(m & ((1u << lane) - 1));
            for (int w = 0; w < kPlanWarps; ++w) {
                if (w < warp) rank += warp_count[w];
                kept += warp_count[w];
            }
            if (keep) {
                if (fits) list[rank] = b;
                put(k0 + rank, b, t);
            }
            __syncthreads();
        }
        before_k0 = k0;
        k0 += kept;
        count = kept;
        ++t;
    }
    if (threadIdx.x < count) {
        few_seq[threadIdx.x] = candidate(threadIdx.x);
        few_tiles[threadIdx.x] = tiles(few_seq[threadIdx.x]);
    }
    __syncthreads();
    for (int i = warp; i < count; i += kPlanWarps)
        for (int pos = t + lane; pos < few_tiles[i]; pos += 32) {
            int k = k0;
            for (int o = 0; o < count; ++o) k += max(0, min(few_tiles[o], pos) - t) + (o < i && few_tiles[o] > pos);
            put(k, few_seq[i], pos);
        }
}

// Grid of an attention kernel and a block's place in it.  Causal tiles cost what they see and stand in their list from long to short:
// with the heads on x, all heads of a tile start before the next tile, and the long ones of every head first (with the tiles on x,
// a head after the other, the last heads' long tiles started when most SMs were done: 28 heads x 1020, forward 69.6 us, backward
// 137; 65 and 122 in this order).  Without a mask all tiles cost the same, and a head's tiles stay together for its keys' sake.
__device__ __forceinline__ unsigned tile_of(int heads_first) { return heads_first ? blockIdx.y : blockIdx.x; }
__device__ __forceinline__ unsigned head_of(int heads_first) { return heads_first ? blockIdx.x : blockIdx.y; }
inline int heads_go_first(int causal, int max_tiles) { return causal && max_tiles <= 65535; }      // the limit of a grid's y
inline dim3 attention_grid(int heads_first, int max_tiles, int heads) {
    return heads_first ? dim3(heads, max_tiles) : dim3(max_tiles, heads);
}

// ------------------------------------------------------------------------------------------ TMA
__device__ __forceinline__ void prefetch_tmap(const CUtensorMap* m) {
    asm volatile("prefetch.tensormap [%0];" ::"l"((uint64_t)m) : "memory");
}
__device__ __forceinline__ void tma_load_2d(void* dst, const CUtensorMap* m, uint64_t* bar, int x, int y) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
        ::"r"(smem_u32(dst)), "l"((uint64_t)m), "r"(smem_u32(bar)), "r"(x), "r"(y)
        : "memory");
}
__device__ __forceinline__ void tma_load_3d(void* dst, const CUtensorMap* m, uint64_t* bar, int x, int y, int z) {
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];"
        ::"r"(smem_u32(dst)), "l"((uint64_t)m), "r"(smem_u32(bar)), "r"(x), "r"(y), "r"(z)
        : "memory");
}
// CTA of a pair: into its own shared memory; the bytes are counted on a barrier of either CTA (`bar`: its cluster address)
__device__ __forceinline__ void tma_load_2d_pair(void* dst, const CUtensorMap* m, uint32_t bar, int x, int y) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes.cta_group::2 [%0], [%1, {%3, %4}], [%2];"
        ::"r"(smem_u32(dst)), "l"((uint64_t)m), "r"(bar), "r"(x), "r"(y)
        : "memory");
}
__device__ __forceinline__ void tma_store_2d(const CUtensorMap* m, const void* src, int x, int y) {
    asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.tile.bulk_group [%0, {%2, %3}], [%1];" ::"l"((uint64_t)m),
                 "r"(smem_u32(src)), "r"(x), "r"(y)
                 : "memory");
}
__device__ __forceinline__ void tma_store_3d(const CUtensorMap* m, const void* src, int x, int y, int z) {
    asm volatile("cp.async.bulk.tensor.3d.global.shared::cta.tile.bulk_group [%0, {%2, %3, %4}], [%1];" ::"l"((uint64_t)m),
                 "r"(smem_u32(src)), "r"(x), "r"(y), "r"(z)
                 : "memory");
}
__device__ __forceinline__ void tma_commit() { asm volatile("cp.async.bulk.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void tma_wait_read() {
    asm volatile("cp.async.bulk.wait_group.read %0;" ::"n"(N) : "memory");
}
template <int N>
__device__ __forceinline__ void tma_wait_all() {
    asm volatile("cp.async.bulk.wait_group %0;" ::"n"(N) : "memory");
}

// ------------------------------------------------------------------------------------------ TMEM
__device__ __forceinline__ void tmem_alloc(uint32_t* dst_smem, uint32_t ncols) {  // whole warp
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(dst_smem)), "r"(ncols)
                 : "memory");
}
__device__ __forceinline__ void tmem_relinquish() {
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols) {  // whole warp
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
// the same for a pair: one warp of each of its CTAs takes part
__device__ __forceinline__ void tmem_alloc_pair(uint32_t* dst_smem, uint32_t ncols) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(dst_smem)), "r"(ncols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc_pair(uint32_t taddr, uint32_t ncols) {
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
__device__ __forceinline__ void fence_before_sync() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_after_sync() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tmem_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tmem_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

// 32 lanes x 32 consecutive fp32 columns: thread i of the warp gets lane (base_lane + i).
__device__ __forceinline__ void tmem_ld_32x32(uint32_t taddr, uint32_t* r) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
        "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
          "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]),
          "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),
          "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr)
        : "memory");
}
__device__ __forceinline__ void tmem_ld_32x16(uint32_t taddr, uint32_t* r) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
          "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr)
        : "memory");
}
__device__ __forceinline__ void tmem_st_32x32(uint32_t taddr, const uint32_t* r) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
        "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, "
        "%17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, %32};"
        ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]),
          "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(r[16]), "r"(r[17]),
          "r"(r[18]), "r"(r[19]), "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]), "r"(r[24]), "r"(r[25]), "r"(r[26]),
          "r"(r[27]), "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31])
        : "memory");
}

__device__ __forceinline__ void tmem_st_32x16(uint32_t taddr, const uint32_t* r) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], "
        "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};"
        ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]),
          "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
        : "memory");
}

// ------------------------------------------------------------------------------------------ UMMA
// Shared-memory matrix descriptor, 128-byte swizzle.  Both majors use 8-row x 128-byte atoms
// (1024 B); `sbo`/`lbo` are byte strides:
//   K-major : rows = M/N index, 128 B = 64 elements of K.  sbo = stride between 8-row groups (1024),
//             lbo unused (1).
//   MN-major: rows = K index, 128 B = 64 elements of M/N.  sbo = stride between 8-K groups (1024),
//             lbo = stride between 64-element M/N atoms.
__device__ __forceinline__ uint64_t smem_desc_sw128(uint32_t saddr, uint32_t lbo_bytes, uint32_t sbo_bytes) {
    uint64_t d = 0;
    d |= (uint64_t)((saddr & 0x3FFFF) >> 4);
    d |= (uint64_t)((lbo_bytes >> 4) & 0x3FFF) << 16;
    d |= (uint64_t)((sbo_bytes >> 4) & 0x3FFF) << 32;
    d |= (uint64_t)1 << 46;  // descriptor version for sm_100
    d |= (uint64_t)2 << 61;  // SWIZZLE_128B
    return d;
}

// Instruction descriptor for kind::f16 with bf16 inputs and fp32 accumulation.
__host__ __device__ constexpr uint32_t idesc_bf16(int M, int N, int a_mn_major, int b_mn_major) {
    return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)a_mn_major << 15) | ((uint32_t)b_mn_major << 16) |
           ((uint32_t)(N >> 3) << 17) | ((uint32_t)(M >> 4) << 24);
}

// D[tmem] (+)= A[smem] * B[smem]; issued by ONE thread.
__device__ __forceinline__ void mma_ss(uint32_t tmem_d, uint64_t desc_a, uint64_t desc_b, uint32_t idesc, uint32_t accum) {
    asm volatile(
        "{\n"
        ".reg .pred p;\n"
        "setp.ne.b32 p, %4, 0;\n"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n"
        "}\n" ::"r"(tmem_d), "l"(desc_a), "l"(desc_b), "r"(idesc), "r"(accum)
        : "memory");
}
// D[tmem] (+)= A[tmem] * B[smem]
__device__ __forceinline__ void mma_ts(uint32_t tmem_d, uint32_t tmem_a, uint64_t desc_b, uint32_t idesc, uint32_t accum) {
    asm volatile(
        "{\n"
        ".reg .pred p;\n"
        "setp.ne.b32 p, %4, 0;\n"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n"
        "}\n" ::"r"(tmem_d), "r"(tmem_a), "l"(desc_b), "r"(idesc), "r"(accum)
        : "memory");
}
// Pair: D has 256 rows, 128 in each CTA's tensor memory; each CTA holds its 128 rows of A and half of the rows of B at the same shared
// addresses.  Issued by ONE thread of the CTA of rank 0.
__device__ __forceinline__ void mma_ss_pair(uint32_t tmem_d, uint64_t desc_a, uint64_t desc_b, uint32_t idesc, uint32_t accum) {
    asm volatile(
        "{\n"
        ".reg .pred p;\n"
        "setp.ne.b32 p, %4, 0;\n"
        "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n"
        "}\n" ::"r"(tmem_d), "l"(desc_a), "l"(desc_b), "r"(idesc), "r"(accum)
        : "memory");
}
// Arrive on the barrier at this address in both CTAs once the MMAs issued so far have completed.
__device__ __forceinline__ void mma_commit_pair(uint64_t* bar) {
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(smem_u32(bar)),
                 "h"((uint16_t)3)
                 : "memory");
}
// Arrive on an mbarrier once all previously issued MMAs of this thread have completed.
__device__ __forceinline__ void mma_commit(uint64_t* bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}

}  // namespace tc05

// ------------------------------------------------------------------------------------------ host: tensor maps
#include <cudaTypedefs.h>
#include <stdio.h>
namespace tc05 {
inline PFN_cuTensorMapEncodeTiled_v12000 encode_fn() {
    static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
    if (!fn) {
        cudaDriverEntryPointQueryResult q;
        void* p = nullptr;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = (PFN_cuTensorMapEncodeTiled_v12000)p;
    }
    return fn;
}
// The encode call is a driver call: on a thread that has made no runtime call yet (an autograd worker whose first op is a
// tensor-core kernel) there is no current context.  cudaFree(nullptr) binds the thread's device's primary one.
template <class F>
inline int encode_with_context(F encode) {
    CUresult r = encode();
    if (r == CUDA_ERROR_INVALID_CONTEXT && cudaFree(nullptr) == cudaSuccess) r = encode();
    return (int)r;
}
// 2-D bf16 tensor [rows, cols] with `ld` elements between rows; box = [box_rows, box_cols]; 128B swizzle.
inline int make_tmap_2d(CUtensorMap* m, const void* base, uint64_t rows, uint64_t cols, uint64_t ld, uint32_t box_rows,
                        uint32_t box_cols, CUtensorMapSwizzle sw = CU_TENSOR_MAP_SWIZZLE_128B) {
    auto fn = encode_fn();
    if (!fn) return -100;
    cuuint64_t dims[2] = {cols, rows};
    cuuint64_t strides[1] = {ld * 2};
    cuuint32_t box[2] = {box_cols, box_rows};
    cuuint32_t es[2] = {1, 1};
    return encode_with_context([&] {
        return fn(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base), dims, strides, box, es,
                  CU_TENSOR_MAP_INTERLEAVE_NONE, sw, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    });
}
// 3-D bf16 tensor [d2, d1, d0] (d0 innermost, contiguous) with element strides s1, s2.
inline int make_tmap_3d(CUtensorMap* m, const void* base, uint64_t d0, uint64_t d1, uint64_t d2, uint64_t s1,
                        uint64_t s2, uint32_t b0, uint32_t b1, uint32_t b2,
                        CUtensorMapSwizzle sw = CU_TENSOR_MAP_SWIZZLE_128B) {
    auto fn = encode_fn();
    if (!fn) return -100;
    cuuint64_t dims[3] = {d0, d1, d2};
    cuuint64_t strides[2] = {s1 * 2, s2 * 2};
    cuuint32_t box[3] = {b0, b1, b2};
    cuuint32_t es[3] = {1, 1, 1};
    return encode_with_context([&] {
        return fn(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(base), dims, strides, box, es,
                  CU_TENSOR_MAP_INTERLEAVE_NONE, sw, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    });
}
// ---- kernels that split their registers between warpgroups
// `regs`: what the warpgroups of a block claim by setmaxnreg, in all.  A claim above the launch's own would wait for good, so such a build
// is refused here.
template <class K>
inline int opt_in(K kern, int smem, int threads, int regs) {
    cudaFuncAttributes a;
    cudaError_t e = cudaFuncGetAttributes(&a, kern);
    if (e != cudaSuccess) return (int)e;
    if (a.numRegs * threads < regs) return -101;
    return (int)cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
}
}  // namespace tc05
