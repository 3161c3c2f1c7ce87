// Persistent, warp-specialised bf16 GEMM on the 5th-gen tensor cores.
//
//   C[M,N] (bf16) = op(A) * op(B) (+ bias[N])        fp32 accumulation in TMEM
//
// Operand layouts (both row-major in memory):
//   A_MN = 0: A is [M, K] (K contiguous)      A_MN = 1: A is stored as [K, M] (M contiguous)
//   B_MN = 0: B is [N, K] (K contiguous)      B_MN = 1: B is stored as [K, N] (N contiguous)
// so forward  y = x W^T      is (A_MN=0, B_MN=0) on (x [T,K], W [N,K]),
//    dgrad    dx = dy W      is (A_MN=0, B_MN=1) on (dy [T,N], W [N,K] read as [K'=N, N'=K]),
//    wgrad    dW = dy^T x    is (A_MN=1, B_MN=1) on (dy [T,N] read as [K'=T, M'=N], x [T,K] read as [K'=T, N'=K]).
//
// One CTA per SM, or a pair of CTAs on two SMs (cta_group::2), walks output tiles of 128, 256 or 512 rows x BN.  Roles:
//   warp 0     : TMA producer  (cp.async.bulk.tensor into a multi-stage 128B-swizzled smem ring)
//   warp 1     : MMA issuer    (one thread issues tcgen05.mma, of a pair one thread of its first CTA; tcgen05.commit frees ring slots)
//   warps 4..11: epilogue      (tcgen05.ld TMEM -> registers -> bf16 -> swizzled smem -> TMA store), four warps per accumulator
// Tensor memory holds two accumulators of 128 rows a CTA: of two tiles, so that the epilogue of tile i overlaps the main loop of tile
// i + 1, or (512 rows) the two halves of one tile.  Tiles are visited in groups of 8 to 16 row blocks per N sweep to keep operands in L2.
// All mbarrier waits are bounded (tc05::mbar_wait); a timeout is reported through `status` and the CTA
// unwinds: it lets in-flight copies land, frees its TMEM and returns.
//
// What bounds a large product with a long main loop is the power cap: every tile size keeps the tensor pipe 90 to 96 % busy, at a clock that the
// energy of its operand traffic sets.  A step of 64 of K brings a CTA 48 KB for 128 x 256 (one CTA), 32 KB for the same as half of a 256-row pair,
// and 48 KB for 256 x 256 as half of a 512-row pair: 19.1 / 14.5 GB through L2 for 8192 x 37888 x 3584 with 256 / 512 rows.  Sustained, TFLOP/s, tiles
// of 128 / 256 / 512 rows (cuBLAS): 8192 x 37888 x 3584 1198 / 1350 / 1388 (1356), 8192 x 3584 x 18944 1224 / 1278 / 1344 (1216), 32760 x 5120 x
// 13824 1161 / 1198 / 1309 (1376), 8192 x 3840 x 1280 1075 / 1149 / 1126 (1108).  Groups of 1024 / 2048 / 8192 rows reach 0.90 / 0.94 / - of the rate
// of groups of 4096 on tiles of 256 rows, - / 0.99 / 0.97 on 512 (8192 x 37888 x 3584); single tiles are used for few rows only.
#include "tc05.cuh"

namespace {

using namespace tc05;

constexpr int BM = 128;
constexpr int BK = 64;
constexpr int kGroupThreads = 128;                        // of an epilogue group
constexpr int kThreads = 128 + 2 * kGroupThreads;
// registers of a thread: 168 at launch; the epilogue holds a packed accumulator row, the issuing warps need few
constexpr int kIssueRegs = 72, kEpiRegs = 216;
constexpr int kSmemBudget = 227 * 1024;

// TM: rows of a tile.  128: one CTA;  256 and 512: a pair of CTAs on two SMs, each with half of the rows and, for the operands, half of the
// columns (cta_group::2).
// SHALLOW (depth up to kStaged): the stores take longer than the products, so each epilogue group has two staging slabs, for one operand
// stage less: one store is under way while the next slab is written.  One slab a group / two, us: 152064 x 3584 at depth 128 311 / 227, at 256
// 328 / 320, at 384 419 / 453; 37888 x 3584 at 64 118 / 88, 256 111 / 103, 320 112 / 114; 8192 x 8192 at 64 52 / 40, 256 51 / 49, 320 52 / 54; 3584 x 3584 at
// 64 12.8 / 10.8, 320 15.9 / 15.4.  The gradient of a vocabulary's weight over 310 rows, behind the products that make its operand, is what the
// line at 320 is for: 381 / 372, 350 rows 408 / 423.
template <int BN, int TM, bool SHALLOW = false>
struct Cfg {
    static constexpr bool kPair = TM > BM;
    static constexpr int kHalves = TM == 512 ? 2 : 1;    // accumulators of 128 rows that a tile has in a CTA's tensor memory
    static constexpr int kBRows = kPair ? BN / 2 : BN;   // rows of B in a CTA's shared memory
    static constexpr int kABytes = kHalves * BM * BK * 2;
    static constexpr int kBBytes = kBRows * BK * 2;
    static constexpr int kStageBytes = kABytes + kBBytes;
    static constexpr int kSlabBufs = SHALLOW ? 2 : 1;
    static constexpr int kCBytes = 2 * kSlabBufs * BM * 64 * 2;  // 128x64 bf16 staging slabs of both epilogue groups
    static constexpr int kAux = 1024;                // barriers etc.
    static constexpr int kStages = (kSmemBudget - kCBytes - kAux - 1024) / kStageBytes;
    static constexpr int kSmem = kStages * kStageBytes + kCBytes + kAux + 1024;
    static constexpr int kAhead = kStages < 3 ? kStages : 3;
    static constexpr int kTmemCols = 2 * BN;
};

// ---- which parts of a product are cut along K
// The unit is a block of `rows` x BN outputs, counted in groups of `group` row blocks, column by column.  Blocks from `full` on are summed as
// `parts` stretches of K each, all others in one go: this alone decides the order of an output's fp32 sum, and with it its bits, whatever
// the tiles are that the work is done in.
struct Cut {
    int full = 0, parts = 1;
    int rows = BM, group = 1024 / BM;
};

__host__ __device__ inline void tile_coords(int tile, int m_blocks, int n_blocks, int group_m, int& mb, int& nb) {
    const int per_group = group_m * n_blocks;
    const int g = tile / per_group;
    const int first_m = g * group_m;
    const int gm = group_m < m_blocks - first_m ? group_m : m_blocks - first_m;
    const int r = tile - g * per_group;
    mb = first_m + r % gm;
    nb = r / gm;
}
__host__ __device__ inline int tile_index(int mb, int nb, int m_blocks, int n_blocks, int group_m) {
    const int first_m = mb / group_m * group_m, gm = group_m < m_blocks - first_m ? group_m : m_blocks - first_m;
    return first_m * n_blocks + nb * gm + mb - first_m;
}

// ---- a CTA's (or pair's) list of work
// Tiles of TM rows.  First those that hold an uncut block, each over the whole of K, in groups of `group` row blocks; then, for each of the
// `parts`, those that hold a cut one, in the cut's own order.  A tile with blocks of both kinds is in both lists, and each time only the
// blocks that it is there for are stored.  The uncut blocks are all rows in front of the cut's first group, and that group's columns up to
// where the cut begins: the last group of row blocks is lower from there on.
struct TileList {
    int n_blocks, k_blocks;                  // of tiles
    int group, last, high, low, from;        // the last group starts at row block `last`; it has `high` row blocks up to column `from` and `low` behind
    int head, tail, tail_group;              // row blocks in front of the cut's first group, row blocks from it on, and of a group of them
    int whole, first, cut, parts;            // tiles in one go; first one with a cut block (of the tail's), and how many have one
    int halves;                              // of the tiles in one go, the last ones that are two items of half their rows each (tiles of 512 rows)
};
// One entry of the list.
struct Item {
    int mb, nb;                              // tile
    int kb0, kb1;
    int part;                                // of K, or -1: in one go
    int half;                                // of the rows, or -1: all
};

__host__ __device__ inline TileList make_list(int M, int N, int K, int TM, int BN, const Cut& c, int halves) {
    TileList l;
    const int m_blocks = (M + TM - 1) / TM;
    l.n_blocks = l.from = (N + BN - 1) / BN;
    l.k_blocks = (K + BK - 1) / BK;
    l.group = (TM == BM ? 1024 : 4096) / TM;
    l.head = m_blocks;
    l.first = l.cut = l.tail = 0;
    l.tail_group = c.group * c.rows / TM;
    l.parts = c.parts;
    l.halves = halves;
    int row = 0, uncut = m_blocks;                                // row: where the cut begins in its first group, in units of the cut
    if (c.parts > 1) {
        tile_coords(c.full, (M + c.rows - 1) / c.rows, l.n_blocks, c.group, row, l.from);
        l.head = row / c.group * c.group * c.rows / TM;
        row %= c.group;
        l.tail = m_blocks - l.head;
        const int high = l.tail < l.tail_group ? l.tail : l.tail_group;
        l.first = l.from * high + row * c.rows / TM;
        l.cut = l.tail * l.n_blocks - l.first;
        uncut = l.head + high;
    }
    l.last = uncut > 0 ? (uncut - 1) / l.group * l.group : 0;
    l.high = uncut - l.last;
    l.low = l.head - l.last;
    l.whole = l.last * l.n_blocks + l.from * l.high + (l.n_blocks - l.from) * l.low + (row * c.rows + TM - 1) / TM;
    return l;
}
__host__ __device__ inline int item_count(const TileList& l) { return l.whole + l.halves + l.cut * l.parts; }

__host__ __device__ inline Item item_at(const TileList& l, int i) {
    Item it{0, 0, 0, l.k_blocks, -1, -1};
    if (i >= l.whole + l.halves) {
        // neighbours in the list are neighbouring tiles over the same part of K, so that they share operand tiles in L2
        const int j = i - l.whole;
        it.part = j / l.cut;
        it.kb0 = it.part * l.k_blocks / l.parts;
        it.kb1 = (it.part + 1) * l.k_blocks / l.parts;
        tile_coords(l.first + j - it.part * l.cut, l.tail, l.n_blocks, l.tail_group, it.mb, it.nb);
        it.mb += l.head;
        return it;
    }
    if (i >= l.whole - l.halves && l.halves) {
        it.half = i >= l.whole;
        i -= it.half * l.halves;
    }
    if (i < l.last * l.n_blocks) {
        tile_coords(i, l.last, l.n_blocks, l.group, it.mb, it.nb);
        return it;
    }
    i -= l.last * l.n_blocks;
    if (i < l.from * l.high) {
        it.nb = i / l.high;
        it.mb = l.last + i - it.nb * l.high;
    } else if ((i -= l.from * l.high) < (l.n_blocks - l.from) * l.low) {
        it.nb = i / l.low;
        it.mb = l.last + i - it.nb * l.low;
        it.nb += l.from;
    } else {
        it.nb = l.from;
        it.mb = l.head + i - (l.n_blocks - l.from) * l.low;
    }
    return it;
}

struct Work {
    TileList list;
    Cut cut;
    int M;
};

struct Params {
    int M, N, K;
    const bf16* bias;
    int* status;
    // output routing (fused all-to-all / reduce-scatter push): where a 128 x 64 output slab goes
    //   mode 0: C[m, n] of this GPU
    //   mode 1: column blocks of width `blk` are dealt round-robin to `world` destinations (Ulysses head scatter):
    //           dst = (n / blk) % world, column (n / (blk * world)) * blk + n % blk, row row_off + m
    //   mode 2: row blocks of `blk` rows go to destination m / blk, stored at row rank * blk + m % blk
    //           (every source has its own slot on the destination, which then sums the slots)
    int mode, blk, world, rank, row_off;
    // optional side output: stats[m * n_slots + n / per_slot] += sum over the tile's columns of (bf16-rounded output)^2,
    // i.e. the sum of squares of every output row per column group, taken from the accumulators (a normalisation over
    // the whole row can then be applied after the columns have been scattered to other GPUs)
    float* stats = nullptr;
    int n_slots = 1, per_slot = 0;
    // split tail (see Cut): fp32 sums of the parts go to `ws`
    float* ws = nullptr;
    Work work;                     // (made by the host unless the device counts: the index arithmetic takes 1 - 2 us, longer than a launch is worth)
    // M (or, with `counts_depth`, K) is what `count` on the device says, less `count_base` and at most what is given here; the tail is then
    // planned by the kernel, which leaves {full, parts} in front of the workspace
    const int* count = nullptr;
    int count_base = 0;
    bool counts_depth = false;
    int most_items = 0;            // of the cut blocks, that the workspace has room for
};
constexpr int kPlanBytes = 256;        // in front of the sums in the workspace of such a product
constexpr int kMostRounds = 8;         // of its split items

constexpr int kMaxDst = 8;
struct TMapSet {
    CUtensorMap m[kMaxDst];
};

// ---- split tail ----
// 168 tiles on 148 SMs take two rounds, the second one with 20 CTAs at work.  The tiles behind the last whole round are therefore cut
// along K into `parts` items each, so that ceil(rem * parts / workers) rounds of a 1 / parts tile follow; the items leave fp32 sums in a
// workspace and a second kernel adds them in their order, adds the bias and rounds, exactly once, to bf16.  No worker waits for another.
//
// What is cut, and into how many parts, is what makes a product of 128-row tiles shortest on as many CTAs as there are SMs, 1 part if the gain
// is under 4 us.  It holds for tiles of every size: another order of the fp32 sums is as exact, but its bits are others, and the layers of
// a model carry them on (16 layers: 1.6 % of a prompt's logits).  A 64-deep step of a 128 x 256 tile takes
// 0.44 us (1.4 PFLOP/s over 148 SMs), and no product is over before its operands have come once at 6.2 TB/s: a single row of tiles
// over a large weight is bound by that, and cutting it only adds traffic.  An item's sums are written and read once at about 4 TB/s, a
// further launch and the shorter main loops cost 6 us (fitted to the figures: at 3 us and 5 TB/s 7800 x 1536 x 4608 was split and
// lost 2 us).
// Measured, 128 x 256 tiles, L2 flushed, whole / split: 1421 x 3584 x 18944 (168 tiles) 218 / 151 us, 405 x 3584 x 37888 (56) 216 / 122,
// 8192 x 3584 x 18944 (896) 828 / 776, 3840 x 1280 x 8192 (150) 132 / 91, 1421 x 3584 x 3584 50 / 46.  Left whole for its operands:
// 85 x 25368 x 27344 247 / 279, 126 x 26744 x 24168 251 / 271.
inline Cut split_plan(int M, int N, int K, int BN, int sms) {
    const int tiles = ((M + BM - 1) / BM) * ((N + BN - 1) / BN), kb = (K + BK - 1) / BK, full = tiles / sms, rem = tiles % sms;
    Cut best;
    best.full = tiles;
    if (!rem) return best;
    const double unit = kb * 0.44 * BN / 256, operands = 2.0 * K * ((double)M + N) / 6.2e6;
    auto at_least = [&](double t) { return t > operands ? t : operands; };
    double least = at_least(unit * (full + 1)) - 4.0;
    for (int parts = 2; parts <= 16 && kb / parts >= 4; ++parts) {
        const int rounds = (rem * parts + sms - 1) / sms;
        const double t = at_least(unit * full + unit * rounds / parts) + 6.0 + rem * parts * (BM * BN * 8e-6 / 4.0);
        if (t < least) {
            least = t;
            best.full = tiles - rem;
            best.parts = parts;
        }
    }
    return best;
}

// Time of a 64-deep step of a tile of 256 columns with 128 / 256 / 512 rows, in us: 0.45 / 0.415 / 0.79 (rates of a burst; an SM, or a pair of
// them, works on it); a 512-row tile has 1 us more for filling its ring anew, and so have its halves, which run at the rate of 256 rows.
__host__ __device__ inline float tile_time(int kb, int rows, int BN) {
    return (rows == BM ? kb * 0.45f : rows == 2 * BM ? kb * 0.415f : kb * 0.79f + 1.f) * BN / 256;
}

// Cut and time of a product whose number of rows only the device knows: the tiles themselves are the units, and their own times decide.  Whole
// tiles are counted, so that there is one cut for each number of row blocks.
struct TailPlan {
    float time;
    int full, parts;
};
__host__ __device__ inline TailPlan plan_tail(int M, int N, int K, int BN, int rows, int workers, int most_parts, int most_items) {
    const int kb = (K + BK - 1) / BK, m_blocks = (M + rows - 1) / rows;
    const float operands = 2.f * K * ((float)m_blocks * rows + N) / 6.2e6f;
    auto at_least = [&](float t) { return t > operands ? t : operands; };
    const int tiles = m_blocks * ((N + BN - 1) / BN), full = tiles / workers, rem = tiles % workers;
    const float unit = tile_time(kb, rows, BN);
    const float whole = at_least(unit * (full + (rem ? 1 : 0)));
    TailPlan best{whole, tiles, 1};
    for (int parts = 2; rem && parts <= most_parts && kb / parts >= 4 && rem * parts <= most_items; ++parts) {
        const int rounds = (rem * parts + workers - 1) / workers;
        const float t = at_least(unit * full + unit * rounds / parts) + 6.f + rem * parts * (rows * BN * 8e-6f / 4.f);
        if (t < best.time && t < whole - 4.f) best = {t, tiles - rem, parts};
    }
    return best;
}

// SWIGLU (BN = 256, K-major operands, no bias): B is the fused [2F, K] gate/up weight, p.N = F.  A tile's accumulator holds
// 128 gate columns (weight rows nb*128 ..) next to the 128 up columns of the same features (rows F + nb*128 ..); the
// epilogue writes silu(gate) * up, so the [M, 2F] pre-activation never reaches memory.
// COUNTED: M, or the depth, is what Params::count says.
template <int BN, bool A_MN, bool B_MN, bool SWIGLU = false, int TM = BM, bool SHALLOW = false, bool COUNTED = false>
__global__ void __launch_bounds__(kThreads, 1)
gemm_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
            const __grid_constant__ TMapSet tmC, Params p) {
    using C = Cfg<BN, TM, SHALLOW>;
    constexpr bool PAIR = C::kPair;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint8_t* sA = smem;
    uint8_t* sB = smem + C::kStages * C::kABytes;
    uint8_t* sC = sB + C::kStages * C::kBBytes;
    uint64_t* full = reinterpret_cast<uint64_t*>(sC + C::kCBytes);
    uint64_t* empty = full + C::kStages;
    uint64_t* tfull = empty + C::kStages;
    uint64_t* tempty = tfull + 2;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(tempty + 2);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
    volatile int* epi_stop = abort_flag + 1;

    const int warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;
    // a worker: this CTA, or the pair that it belongs to
    const int rank = PAIR ? (int)cluster_rank() : 0;
    const int worker = PAIR ? blockIdx.x / 2 : blockIdx.x, n_workers = PAIR ? gridDim.x / 2 : gridDim.x;
    if (threadIdx.x == 0) {
        for (int s = 0; s < C::kStages; ++s) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], 1);
        }
        for (int a = 0; a < 2; ++a) {
            mbar_init(&tfull[a], 1);
            mbar_init(&tempty[a], (PAIR ? 2 : 1) * kGroupThreads / 32);
        }
        *abort_flag = 0;
        fence_barrier_init();
        prefetch_tmap(&tmA);
        prefetch_tmap(&tmB);
        for (int d = 0; d < (p.mode ? p.world : 1); ++d) prefetch_tmap(&tmC.m[d]);
    }
    if (warp == 1) {
        if constexpr (PAIR) {
            tmem_alloc_pair(tmem_slot, C::kTmemCols);
        } else {
            tmem_alloc(tmem_slot, C::kTmemCols);
            tmem_relinquish();
        }
    }
    fence_before_sync();
    __syncthreads();
    if constexpr (PAIR) cluster_sync();          // the other CTA's barriers are there, too
    fence_after_sync();
    const uint32_t tmem_base = *tmem_slot;
    wait_for_predecessor();
    let_successor_start();

    Work& counted = *reinterpret_cast<Work*>(tmem_slot + 4);
    if constexpr (COUNTED) {
        if (threadIdx.x == 0) {
            const int n = max(0, *p.count - p.count_base);
            Work w = p.work;
            if (p.counts_depth) p.K = min(p.K, n);
            else w.M = min(p.M, n);
            if (p.ws != nullptr && !p.counts_depth) {
                const TailPlan t = plan_tail(w.M, p.N, p.K, BN, TM, n_workers, 16, p.most_items);
                w.cut.full = t.full;
                w.cut.parts = t.parts;
                if (blockIdx.x == 0) {
                    int* plan = reinterpret_cast<int*>(p.ws - kPlanBytes / 4);
                    plan[0] = t.full;
                    plan[1] = t.parts;
                }
            }
            w.list = make_list(w.M, p.N, p.K, TM, BN, w.cut, 0);
            counted = w;
        }
        __syncthreads();
    }
    const Work& work = COUNTED ? counted : p.work;          // (in shared memory: registers for it would be spilled)
    const TileList& list = work.list;
    const int n_items = item_count(list);

    if (warp < 4) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kIssueRegs));
        if (warp == 0) {
        // ------------------------------------------------------------------ TMA producer
        if (lane == 0) {
            int stage = 0;
            uint32_t phase = 0;
            bool ok = true;
            for (int i = worker; i < n_items && ok; i += n_workers) {
                const Item item = item_at(list, i);
                const int mb = item.mb, nb = item.nb;
                for (int kb = item.kb0; kb < item.kb1; ++kb) {
                    if (!mbar_wait(&empty[stage], phase ^ 1, abort_flag)) {
                        atomicExch(p.status, MM_TIMEOUT_TMA);
                        ok = false;
                        break;
                    }
                    uint8_t* a = sA + stage * C::kABytes;
                    uint8_t* b = sB + stage * C::kBBytes;
                    const int m0 = mb * TM + rank * (TM / 2), n0 = nb * BN + rank * C::kBRows;
                    const uint32_t bar = PAIR ? cluster_addr(&full[stage], 0) : 0;
                    auto load = [&](uint8_t* dst, const CUtensorMap* m, int x, int y) {
                        if constexpr (PAIR) tma_load_2d_pair(dst, m, bar, x, y);
                        else tma_load_2d(dst, m, &full[stage], x, y);
                    };
                    // (a pair's copies are all counted in the CTA of rank 0, where the products are issued)
                    if (rank == 0) mbar_expect_tx(&full[stage], C::kStageBytes * (PAIR ? 2 : 1));
                    if constexpr (!A_MN) {
                        load(a, &tmA, kb * BK, m0);
                    } else {
#pragma unroll
                        for (int j = 0; j < C::kHalves * BM / 64; ++j) load(a + j * (BK * 128), &tmA, m0 + j * 64, kb * BK);
                    }
                    if constexpr (SWIGLU && PAIR) {
                        load(b, &tmB, kb * BK, rank * p.N + nb * 128);
                    } else if constexpr (SWIGLU) {
                        load(b, &tmB, kb * BK, nb * 128);
                        load(b + 128 * 128, &tmB, kb * BK, p.N + nb * 128);
                    } else if constexpr (!B_MN) {
                        load(b, &tmB, kb * BK, n0);
                    } else {
#pragma unroll
                        for (int j = 0; j < C::kBRows / 64; ++j) load(b + j * (BK * 128), &tmB, n0 + j * 64, kb * BK);
                    }
                    if (++stage == C::kStages) {
                        stage = 0;
                        phase ^= 1;
                    }
                }
            }
            if constexpr (PAIR)                  // every slot's release, which comes from the other CTA, has arrived before this one ends
                for (int s = 0; s < C::kStages && ok; ++s) {
                    ok = mbar_wait(&empty[stage], phase ^ 1, abort_flag);
                    if (++stage == C::kStages) {
                        stage = 0;
                        phase ^= 1;
                    }
                }
        }
        } else if (warp == 1) {
        // ------------------------------------------------------------------ MMA issuer
        if (lane == 0 && rank == 0) {
            constexpr uint32_t idesc = idesc_bf16(PAIR ? 2 * BM : BM, BN, A_MN ? 1 : 0, B_MN ? 1 : 0);
            int stage = 0;
            uint32_t phase = 0;
            int used0 = 0, used1 = 0;               // items that each accumulator has had
            bool ok = true;
            auto step = [](int& s, uint32_t& ph) {
                if (++s == C::kStages) {
                    s = 0;
                    ph ^= 1;
                }
            };
            auto arrived = [&](int s, uint32_t ph) {
                if (mbar_wait(&full[s], ph, abort_flag)) return true;
                atomicExch(p.status, MM_TIMEOUT_MMA);
                return ok = false;
            };
            auto drained = [&](int acc) {
                const uint32_t parity = ((acc ? used1 : used0) & 1) ^ 1;
                ++(acc ? used1 : used0);
                if (PAIR ? mbar_wait_cluster(&tempty[acc], parity, abort_flag) : mbar_wait(&tempty[acc], parity, abort_flag)) {
                    fence_after_sync();
                    return true;
                }
                atomicExch(p.status, MM_TIMEOUT_MMA);
                return ok = false;
            };
            auto done = [&](uint64_t* bar) {
                if constexpr (PAIR) mma_commit_pair(bar);
                else mma_commit(bar);
            };
            // products of one slot's operands; h: which 128 rows of the CTA's A tile
            auto products = [&](int s, int h, int acc, bool first) {
                fence_after_sync();
                const uint32_t a0 = smem_u32(sA + s * C::kABytes) + h * BM * BK * 2;
                const uint32_t b0 = smem_u32(sB + s * C::kBBytes);
#pragma unroll
                for (int k = 0; k < BK / 16; ++k) {
                    // K-major: 16 elements of K = 32 bytes inside the swizzle atom.
                    // MN-major: 16 rows of K = two 8-row groups = 2048 bytes.
                    const uint64_t da = A_MN ? smem_desc_sw128(a0 + k * 2048, BK * 128, 1024)
                                             : smem_desc_sw128(a0 + k * 32, 16, 1024);
                    const uint64_t db = B_MN ? smem_desc_sw128(b0 + k * 2048, BK * 128, 1024)
                                             : smem_desc_sw128(b0 + k * 32, 16, 1024);
                    const uint32_t accum = !first || k ? 1u : 0u;
                    if constexpr (PAIR) mma_ss_pair(tmem_base + acc * BN, da, db, idesc, accum);
                    else mma_ss(tmem_base + acc * BN, da, db, idesc, accum);
                }
            };
            int it = 0;
            for (int i = worker; i < n_items && ok; i += n_workers, ++it) {
                const Item item = item_at(list, i);
                auto alone = [&](int h, int acc) {           // an item with one accumulator
                    if (!drained(acc)) return;
                    for (int kb = item.kb0; kb < item.kb1 && arrived(stage, phase); ++kb) {
                        products(stage, h, acc, kb == item.kb0);
                        done(&empty[stage]);        // slot reusable once these MMAs have read it
                        step(stage, phase);
                    }
                    if (ok) done(&tfull[acc]);
                };
                if constexpr (C::kHalves == 1) {
                    alone(0, it & 1);
                } else if (item.half >= 0) {
                    alone(item.half, item.half);
                } else {
                    // Tensor memory holds one tile, so its first accumulator runs ahead of the second at both ends, by up to kAhead
                    // slots: it is complete, and drained, while the second one's last products run, and the next tile starts on it
                    // while the second one is drained.
                    const int n = item.kb1 - item.kb0, head = min(n, C::kAhead), tail = min(n - head, C::kAhead);
                    auto ahead = [&](int count, bool first, bool last) {
                        int s = stage;
                        uint32_t ph = phase;
                        if (first && !drained(0)) return;
                        for (int k = 0; k < count; ++k) {
                            if (!arrived(s, ph)) return;
                            products(s, 0, 0, first && k == 0);
                            step(s, ph);
                        }
                        if (last) done(&tfull[0]);
                        if (first && !drained(1)) return;
                        for (int k = 0; k < count; ++k) {
                            products(stage, 1, 1, first && k == 0);
                            done(&empty[stage]);
                            step(stage, phase);
                        }
                        if (last) done(&tfull[1]);
                    };
                    ahead(head, true, head == n);
                    for (int k = head; k < n - tail && ok && arrived(stage, phase); ++k) {
                        products(stage, 0, 0, false);
                        products(stage, 1, 1, false);
                        done(&empty[stage]);
                        step(stage, phase);
                    }
                    if (ok && tail) ahead(tail, false, true);
                }
            }
        }
        }
    } else {
        asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kEpiRegs));
        // ------------------------------------------------------------------ epilogue
        // Group g drains accumulator g.  A thread takes its whole row into registers, as bf16, before anything is stored: the products
        // of the next tile wait for nothing but these reads.
        const int q = warp & 3;            // TMEM lane quarter this warp may read
        const int row = q * 32 + lane;     // row inside the 128-row tile
        const int group = (warp >> 2) - 1;
        const bool issuer = threadIdx.x % kGroupThreads == 0;
        uint8_t* bufs = sC + group * C::kSlabBufs * (BM * 128);
        auto group_sync = [&] { asm volatile("bar.sync %0, 128;" ::"r"(1 + group) : "memory"); };
        auto drained = [&] {
            fence_before_sync();
            __syncwarp();
            if (lane == 0) {
                if constexpr (PAIR) mbar_arrive_cluster(cluster_addr(&tempty[group], 0));
                else mbar_arrive(&tempty[group]);
            }
        };
        const uint32_t t_row = tmem_base + group * BN + ((uint32_t)(q * 32) << 16);
        const bool wide_bias = (reinterpret_cast<uintptr_t>(p.bias) & 15) == 0;
        constexpr int kSlabs = SWIGLU ? 2 : BN / 64;         // of 64 output columns
        int it = 0, use = 0;
        for (int i = worker; i < n_items; i += n_workers, ++it) {
            if (C::kHalves == 1 && (it & 1) != group) continue;
            const Item item = item_at(list, i);
            if (C::kHalves == 2 && item.half >= 0 && item.half != group) continue;
            const int mb = item.mb, nb = item.nb;
            const int h = C::kHalves == 1 ? 0 : group, m0 = mb * TM + rank * (TM / 2) + h * BM;
            bool mine = m0 < work.M;                      // these 128 rows are what the item is there for
            size_t slot = 0;                              // of the workspace, in blocks of 128 rows
            if (!SWIGLU && list.cut > 0 && mine) {
                const Cut& cut = work.cut;
                const int c = tile_index(m0 / cut.rows, nb, (work.M + cut.rows - 1) / cut.rows, list.n_blocks, cut.group) - cut.full;
                mine = (item.part >= 0) == (c >= 0);
                if (item.part >= 0 && mine) slot = (size_t)(c * cut.parts + item.part) * (cut.rows / BM) + m0 % cut.rows / BM;
            }
            if (!mbar_wait(&tfull[group], use++ & 1, abort_flag) && lane == 0) atomicExch(p.status, MM_TIMEOUT_EPI);
            __syncwarp();
            fence_after_sync();
            const bool none = item.kb0 == item.kb1;       // of a product without depth: nothing was accumulated
            uint32_t v[kSlabs * 32];
            if (!SWIGLU && item.part >= 0) {
                // [column / 4][row][4]: the lanes of a warp write neighbouring rows of a column group
                float4* dst = reinterpret_cast<float4*>(p.ws) + slot * (BM * BN / 4) + row;
#pragma unroll 1
                for (int slab = 0; slab < kSlabs; ++slab) {
                    uint32_t r[64];
                    tmem_ld_32x32(t_row + slab * 64, r);
                    tmem_ld_32x32(t_row + slab * 64 + 32, r + 32);
                    tmem_wait_ld();
                    if (slab == kSlabs - 1) drained();
                    if (none)
#pragma unroll
                        for (int c = 0; c < 64; ++c) r[c] = 0;
                    if (mine)
#pragma unroll
                        for (int c = 0; c < 16; ++c)
                            dst[(slab * 16 + c) * BM] = make_float4(__uint_as_float(r[4 * c]), __uint_as_float(r[4 * c + 1]),
                                                                    __uint_as_float(r[4 * c + 2]), __uint_as_float(r[4 * c + 3]));
                }
            } else {
#pragma unroll
                for (int slab = 0; slab < kSlabs; ++slab) {
                    uint32_t r[64];
                    const int n0 = (SWIGLU ? nb * 128 : nb * BN) + slab * 64;
                    if constexpr (SWIGLU) {
#pragma unroll
                        for (int half = 0; half < 2; ++half) {
                            uint32_t u[32];
                            tmem_ld_32x32(t_row + slab * 64 + half * 32, r + half * 32);
                            tmem_ld_32x32(t_row + 128 + slab * 64 + half * 32, u);
                            tmem_wait_ld();
#pragma unroll
                            for (int c = 0; c < 32; ++c) {
                                const float g = __uint_as_float(r[half * 32 + c]);
                                r[half * 32 + c] = __float_as_uint(__fdividef(g, 1.f + __expf(-g)) * __uint_as_float(u[c]));
                            }
                        }
                    } else {
                        tmem_ld_32x32(t_row + slab * 64, r);
                        tmem_ld_32x32(t_row + slab * 64 + 32, r + 32);
                        tmem_wait_ld();
                    }
                    if (slab == kSlabs - 1) drained();
                    if (none)
#pragma unroll
                        for (int c = 0; c < 64; ++c) r[c] = 0;
                    if (!SWIGLU && p.bias != nullptr) {
                        if (wide_bias && n0 + 64 <= p.N) {
#pragma unroll
                            for (int c = 0; c < 64; c += 8) {
                                float b[8];
                                unpack8(*reinterpret_cast<const Vec8*>(p.bias + n0 + c), b);
#pragma unroll
                                for (int e = 0; e < 8; ++e) r[c + e] = __float_as_uint(__uint_as_float(r[c + e]) + b[e]);
                            }
                        } else {
#pragma unroll
                            for (int c = 0; c < 64; ++c) {
                                const int n = n0 + c;
                                const float bv = n < p.N ? __bfloat162float(p.bias[n]) : 0.f;
                                r[c] = __float_as_uint(__uint_as_float(r[c]) + bv);
                            }
                        }
                    }
                    if (!SWIGLU && p.stats != nullptr) {
                        float ss = 0.f;
#pragma unroll
                        for (int c = 0; c < 64; ++c) {
                            const float x = __bfloat162float(__float2bfloat16_rn(__uint_as_float(r[c])));
                            ss += (n0 + c < p.N) ? x * x : 0.f;
                        }
                        const int m = m0 + row;
                        if (m < p.M && n0 < p.N) atomicAdd(&p.stats[(size_t)m * p.n_slots + n0 / p.per_slot], ss);
                    }
#pragma unroll
                    for (int c = 0; c < 32; ++c) {
                        const bf162 t = __floats2bfloat162_rn(__uint_as_float(r[2 * c]), __uint_as_float(r[2 * c + 1]));
                        v[slab * 32 + c] = *reinterpret_cast<const uint32_t*>(&t);
                    }
                }
            }
            // one go / no-go decision for all threads of the group before its barriers below
            group_sync();
            if (issuer) epi_stop[group] = *abort_flag;
            group_sync();
            if (epi_stop[group]) break;
            if (!SWIGLU && item.part >= 0) continue;
#pragma unroll
            for (int slab = 0; slab < kSlabs; ++slab) {
                const int n0 = (SWIGLU ? nb * 128 : nb * BN) + slab * 64;
                uint8_t* buf = bufs + slab % C::kSlabBufs * (BM * 128);
                if (issuer) tma_wait_read<C::kSlabBufs - 1>();      // the store that last read this buffer has drained
                group_sync();
#pragma unroll
                for (int c = 0; c < 8; ++c)
                    *reinterpret_cast<uint4*>(buf + row * 128 + ((c ^ (row & 7)) << 4)) =
                        make_uint4(v[slab * 32 + 4 * c], v[slab * 32 + 4 * c + 1], v[slab * 32 + 4 * c + 2], v[slab * 32 + 4 * c + 3]);
                fence_proxy_async();
                group_sync();
                if (issuer) {
                    if (p.mode == 0) {
                        if (mine && n0 < p.N) tma_store_2d(&tmC.m[0], buf, n0, m0);
                    } else if (p.mode == 1) {
                        const int b = n0 / p.blk;
                        tma_store_2d(&tmC.m[b % p.world], buf, (b / p.world) * p.blk + n0 % p.blk, p.row_off + m0);
                    } else {
                        tma_store_2d(&tmC.m[m0 / p.blk], buf, n0, p.rank * p.blk + m0 % p.blk);
                    }
                    tma_commit();
                }
            }
        }
        if (issuer) tma_wait_all<0>();
    }

    // ---------------------------------------------------------------------- teardown
    if (*abort_flag) {
        // give copies that may still be in flight time to land before the CTA's smem is released
        for (int i = 0; i < 64; ++i) __nanosleep(1000);
    }
    fence_before_sync();
    __syncthreads();
    if constexpr (PAIR) cluster_sync();          // nothing of the other CTA reaches for this one's memory from here on
    if (warp == 1) {
        fence_after_sync();
        if constexpr (PAIR) tmem_dealloc_pair(tmem_base, C::kTmemCols);
        else tmem_dealloc(tmem_base, C::kTmemCols);
    }
}

// ---- choice of the tile ----
struct Plan {
    int rows;              // of a tile
    Cut cut;
    int halves;            // see TileList::halves
    float time;            // estimated, us
    int most_items = 0;    // see Params::most_items
    bool staged = false;   // two staging slabs an epilogue group, see Cfg
};

// Depth up to which tiles are one CTA's: the accumulators are emptied and written as long as the next tile's products take, or longer, and
// a CTA of a pair waits for both of its halves.  152064 x 3584, 128 / 256 / 512 rows: depth 256 299 / 339 / 342 us, 384 388 / 400 / 411,
// 448 429 / 394 / 445; 8192 x 8192: 256 47 / 55 / 55, 384 53 / 57 / 61, 448 59 / 59 / 65; 3584 x 3584: 64 17 / 21 / 24, 384 21.5 / 23.5 / 27.
constexpr int kShallow = 6 * BK, kStaged = 5 * BK;

// Time of a product on tiles of `rows` rows, in us.  The list is dealt out one by one: the CTA
// with the most work has the last tile in one go, or is the first behind it.
inline Plan plan_tiles(int M, int N, int K, int BN, int rows, int workers, const Cut& cut) {
    const int kb = (K + BK - 1) / BK;
    const float unit = tile_time(kb, rows, BN), operands = 2.f * K * ((float)M + N) / 6.2e6f;
    const TileList l = make_list(M, N, K, rows, BN, cut, 0);
    const int q = l.whole / workers, r = l.whole % workers, parts = l.cut * l.parts;
    Plan p{rows, cut, 0, 0.f};
    if (l.cut) {
        const int each = parts / workers, more = parts % workers;        // parts go to the CTAs from number r on
        const float first = r ? q + 1 + (float)(each + (more > workers - r)) / l.parts : 0.f;
        const float other = q + (float)(each + (more > 0)) / l.parts;
        p.time = unit * (first > other ? first : other);
    } else {
        p.time = unit * (q + (r > 0));
        // 512 rows: the last tiles as two halves each, where these fit one round.  152 tiles on 74 pairs (4096 x 4864 x 2568) 101.4 us whole,
        // 99.3 with halves, 101.4 on tiles of 256 rows; behind one round only 256 rows are faster: 96 tiles (3626 x 2992 x 3880) 93.2, 91.5, 89.1.
        if (rows == 4 * BM && q >= 2 && r && 2 * r <= workers) {
            p.halves = r;
            p.time = unit * q + tile_time(kb, 2 * BM, BN) + 1.f;
        }
    }
    if (p.time < operands) p.time = operands;
    if (l.cut) p.time += 6.f + (((M + BM - 1) / BM) * l.n_blocks - cut.full) * l.parts * (BM * BN * 8e-6f / 4.f);      // the sums
    return p;
}

// The tile size, of those that M fills more than half of, with the shortest estimate.  device_rows: the device counts the rows, M at most.
inline Plan make_plan(int M, int N, int K, int BN, int sms, bool may_pair, bool may_split, bool device_rows = false) {
    Cut cut;
    if (may_split) cut = split_plan(M, N, K, BN, sms);
    Plan best{BM, cut, 0, 0.f};
    float least = 1e30f;
    for (int rows = BM; rows == BM || (may_pair && K > kShallow && rows <= 4 * BM && M > rows / 2); rows *= 2) {
        const int workers = rows > BM ? sms / 2 : sms;
        Plan p = plan_tiles(M, N, K, BN, rows, workers, cut);
        if (device_rows) {
            p.cut.rows = rows;
            p.cut.group = (rows == BM ? 1024 : 4096) / rows;
            p.cut.parts = 1;                                    // the device's plan takes its place
            p.halves = 0;
            p.time = plan_tail(M, N, K, BN, rows, workers, 16, 1 << 30).time;
        }
        if (p.time < least) {
            least = p.time;
            best = p;
        }
    }
    best.staged = best.rows == BM && BN == 256 && K <= kStaged;
    return best;
}

// bytes of the workspace that the plan's split tiles take (their fp32 sums)
inline long long split_bytes(const Plan& p, int M, int N, int BN) {
    if (p.cut.parts == 1) return 0;
    const long long tiles = (long long)((M + p.cut.rows - 1) / p.cut.rows) * ((N + BN - 1) / BN);
    return (tiles - p.cut.full) * p.cut.parts * p.cut.rows * BN * 4;
}

inline int sm_count() {
    static int sms = 0;
    if (!sms) {
        int dev = 0;
        cudaGetDevice(&dev);
        if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || sms <= 0) sms = 148;
    }
    return sms;
}

// Cut block of C = bf16(sum over the parts of the workspace + bias); a thread makes 8 columns of a row.
// It starts when the product has ended: a product's CTA leaves no registers for a block of it, so that, started early, all its blocks came up on
// the first SMs that fell idle.  Products behind one another, early / not: 1421 x 3584 x 3584 41.1 / 33.4 us, 1421 x 3584 x 18944 155.0 / 145.6,
// 2533 x 5752 x 6480 143.9 / 132.7, 405 x 3584 x 18944 62.5 / 60.2.
template <int BN>
__global__ void __launch_bounds__(256) sum_parts_kernel(const float* __restrict__ ws, bf16* __restrict__ C, const bf16* __restrict__ bias, int M, int N,
                                                        long long ldc, Cut cut, const int* __restrict__ count, int count_base) {
    let_successor_start();
    const int i = blockIdx.x * 256 + threadIdx.x, row = i % BM, cg = i / BM % (BN / 8), sub = i / (BM * BN / 8), t = blockIdx.y;
    int mb, nb;                                                                                   // cg: group of 8 columns
    if (count != nullptr) {
        M = min(M, max(0, *count - count_base));
        cut.full = reinterpret_cast<const int*>(ws)[0];
        cut.parts = reinterpret_cast<const int*>(ws)[1];
        ws += kPlanBytes / 4;
        if (cut.parts == 1 || cut.full + t >= ((M + cut.rows - 1) / cut.rows) * ((N + BN - 1) / BN)) return;
    }
    tile_coords(cut.full + t, (M + cut.rows - 1) / cut.rows, (N + BN - 1) / BN, cut.group, mb, nb);
    const int m = mb * cut.rows + sub * BM + row, n = nb * BN + cg * 8, parts = cut.parts;
    if (m >= M || n >= N) return;
    const size_t step = (size_t)cut.rows * BN / 4;               // between the parts of a block, in float4
    const float4* src = reinterpret_cast<const float4*>(ws) + t * parts * step + (size_t)sub * (BM * BN / 4) + (size_t)(2 * cg) * BM + row;
    float f[8] = {0, 0, 0, 0, 0, 0, 0, 0};
#pragma unroll 4
    for (int q = 0; q < parts; ++q) {
        const float4 a = src[q * step], b = src[q * step + BM];
        f[0] += a.x; f[1] += a.y; f[2] += a.z; f[3] += a.w;
        f[4] += b.x; f[5] += b.y; f[6] += b.z; f[7] += b.w;
    }
    bf16* dst = C + (size_t)m * ldc + n;
    if (n + 8 <= N) {
        if (bias)
#pragma unroll
            for (int k = 0; k < 8; ++k) f[k] += __bfloat162float(bias[n + k]);
        *reinterpret_cast<Vec8*>(dst) = pack8(f);
    } else {
        for (int k = 0; n + k < N; ++k) dst[k] = __float2bfloat16(f[k] + (bias ? __bfloat162float(bias[n + k]) : 0.f));
    }
}

struct Route {
    int mode = 0, blk = 0, world = 1, rank = 0, row_off = 0;
    void* const* dst = nullptr;     // mode != 0: `world` destination base pointers (peer-mapped)
    long long dst_rows = 0, dst_cols = 0;
    float* stats = nullptr;         // see Params::stats
    int n_slots = 1;
    const int* count = nullptr;     // see Params::count
    int count_base = 0;
    bool counts_depth = false;
};

template <int BN, bool A_MN, bool B_MN, bool SWIGLU, int TM, bool SHALLOW = false, bool COUNTED = false>
int launch_tiles(const void* A, const void* B, void* Cc, const void* bias, int M, int N, int K, long long lda, long long ldb,
                 long long ldc, int* status, cudaStream_t st, const Route& rt, const Plan& plan, float* ws) {
    using C = Cfg<BN, TM, SHALLOW>;
    constexpr bool PAIR = C::kPair;
    CUtensorMap tA, tB;
    TMapSet tC;
    int r;
    // A_MN: memory is [K, M] -> rows=K, cols=M, box = 64 k-rows x 64 m ;  else rows=M, cols=K, box = 128 x 64
    r = A_MN ? make_tmap_2d(&tA, A, K, M, lda, BK, 64) : make_tmap_2d(&tA, A, M, K, lda, C::kHalves * BM, BK);
    if (r) return 1000 + r;
    if (SWIGLU)
        r = make_tmap_2d(&tB, B, 2LL * N, K, ldb, 128, BK);      // gate and up halves are fetched as two 128-row boxes
    else
        r = B_MN ? make_tmap_2d(&tB, B, K, N, ldb, BK, 64) : make_tmap_2d(&tB, B, N, K, ldb, C::kBRows, BK);
    if (r) return 2000 + r;
    if (rt.mode == 0) {
        r = make_tmap_2d(&tC.m[0], Cc, M, N, ldc, BM, 64);
        if (r) return 3000 + r;
    } else {
        if (rt.world > kMaxDst) return -5;
        for (int d = 0; d < rt.world; ++d) {
            if (rt.mode == 1) {
                // this launch owns rows [row_off, row_off + M) of every destination: the map covers exactly those, so the
                // last (partial) row tile is clipped instead of spilling into the next source's rows
                if (rt.row_off + (long long)M > rt.dst_rows) return -6;
                r = make_tmap_2d(&tC.m[d], (const char*)rt.dst[d] + (size_t)rt.row_off * ldc * 2, M, rt.dst_cols, ldc, BM, 64);
            } else {
                r = make_tmap_2d(&tC.m[d], rt.dst[d], rt.dst_rows, rt.dst_cols, ldc, BM, 64);
            }
            if (r) return 3000 + r;
        }
    }
    auto kern = gemm_kernel<BN, A_MN, B_MN, SWIGLU, TM, SHALLOW, COUNTED>;
    static bool done = false;
    if (!done) {
        r = opt_in(kern, C::kSmem, kThreads, (kIssueRegs + 2 * kEpiRegs) * 128);
        if (r) return r;
        done = true;
    }
    Params p{M, N, K, (const bf16*)bias, status, rt.mode, rt.blk, rt.world, rt.rank, rt.mode == 1 ? 0 : rt.row_off,
             rt.stats, rt.n_slots, rt.n_slots > 0 ? N / rt.n_slots : N};
    const int workers = PAIR ? sm_count() / 2 : sm_count();
    const bool dynamic_rows = rt.count != nullptr && !rt.counts_depth;
    p.work = {make_list(M, SWIGLU ? 2 * N : N, K, TM, BN, plan.cut, plan.halves), plan.cut, M};
    const int items = item_count(p.work.list);
    if (dynamic_rows) p.ws = ws + kPlanBytes / 4;
    else if (plan.cut.parts > 1) p.ws = ws;
    p.count = rt.count;
    p.count_base = rt.count_base;
    p.counts_depth = rt.counts_depth;
    p.most_items = plan.most_items;
    r = launch_after(kern, PAIR ? 2 : 1, dim3((items < workers && !dynamic_rows ? items : workers) * (PAIR ? 2 : 1)), kThreads, C::kSmem, st, tA, tB, tC, p);
    if (r) return r;
    const int cut = dynamic_rows ? (plan.most_items / 2 < workers ? plan.most_items / 2 : workers - 1)           // blocks, at most
                    : plan.cut.parts > 1 ? ((M + plan.cut.rows - 1) / plan.cut.rows) * ((N + BN - 1) / BN) - plan.cut.full : 0;
    if (cut)
        sum_parts_kernel<BN><<<dim3(plan.cut.rows * BN / 8 / 256, cut), 256, 0, st>>>(ws, (bf16*)Cc, (const bf16*)bias, M, N, ldc, plan.cut,
                                                                                     dynamic_rows ? rt.count : nullptr, rt.count_base);
    return (int)cudaGetLastError();
}

template <int BN, bool A_MN, bool B_MN, bool SWIGLU = false>
int launch(const void* A, const void* B, void* Cc, const void* bias, int M, int N, int K, long long lda, long long ldb,
           long long ldc, int* status, cudaStream_t st, const Route& rt = Route(), float* ws = nullptr, long long ws_bytes = 0) {
    const bool may_pair = BN == 256 && rt.mode == 0, may_split = !SWIGLU && ws && rt.mode == 0;
    const int cols = SWIGLU ? 2 * N : N;                  // a tile of a SwiGLU product: 128 features
    const bool device_rows = rt.count != nullptr && !rt.counts_depth;
    Plan plan = make_plan(M, cols, K, BN, sm_count(), may_pair, may_split, device_rows);
    if (split_bytes(plan, M, cols, BN) > ws_bytes) plan = make_plan(M, cols, K, BN, sm_count(), may_pair, false, device_rows);
    if constexpr (BN == 256 && !SWIGLU && (!A_MN || B_MN))
        if (rt.count != nullptr) {
            plan.halves = 0;
            if (device_rows) plan.most_items = (int)((ws_bytes - kPlanBytes) / (plan.rows * BN * 4));
            if (plan.rows == 512) return launch_tiles<BN, A_MN, B_MN, SWIGLU, 512, false, true>(A, B, Cc, bias, M, N, K, lda, ldb, ldc, status, st, rt, plan, ws);
            if (plan.rows == 256) return launch_tiles<BN, A_MN, B_MN, SWIGLU, 256, false, true>(A, B, Cc, bias, M, N, K, lda, ldb, ldc, status, st, rt, plan, ws);
            return launch_tiles<BN, A_MN, B_MN, SWIGLU, BM, false, true>(A, B, Cc, bias, M, N, K, lda, ldb, ldc, status, st, rt, plan, ws);
        }
    if constexpr (BN == 256) {
        if (plan.rows == 512) return launch_tiles<BN, A_MN, B_MN, SWIGLU, 512>(A, B, Cc, bias, M, N, K, lda, ldb, ldc, status, st, rt, plan, ws);
        if (plan.rows == 256) return launch_tiles<BN, A_MN, B_MN, SWIGLU, 256>(A, B, Cc, bias, M, N, K, lda, ldb, ldc, status, st, rt, plan, ws);
    }
    if constexpr (BN == 256 && !SWIGLU)
        if (plan.staged) return launch_tiles<BN, A_MN, B_MN, SWIGLU, BM, true>(A, B, Cc, bias, M, N, K, lda, ldb, ldc, status, st, rt, plan, ws);
    return launch_tiles<BN, A_MN, B_MN, SWIGLU, BM>(A, B, Cc, bias, M, N, K, lda, ldb, ldc, status, st, rt, plan, ws);
}

}  // namespace

// csrc/decode.cu: products with up to 4 rows
MM_API int mm_gemv_bf16(const void* x, const void* w, const void* bias, const void* norm, const void* res, void* out, int M, int N,
                        int K, long long ldx, long long ldw, long long ldr, long long ldo, float eps, int swiglu, cudaStream_t st);

namespace {
// Up to 4 rows: the weights are streamed once through CUDA cores.  The line lies there because a fifth row makes the fp32
// multiply-adds, not HBM, the limit (8 multiply-adds per weight element and SM cycle at 4 rows), and x has to fit shared memory.
// Four rows are at that limit: where the 128 x 256 tiles of the weight's `rows` rows keep half of the SMs busy, tiles are as fast or
// faster (18944 x 3584: 44 us both ways, 37888 x 3584 67 against 73, 152064 x 3584 198 against 243; 8192 x 8192 64 against 56;
// three rows 202 against 195 at 152064 x 3584).
bool skinny(int M, int rows, int K) {
    return M <= 4 && rows % 2 == 0 && K % 8 == 0 && (long long)M * K <= 80 * 1024 && (M < 4 || rows < 74 * 256);
}
}  // namespace

// Rows of the tiles that mm_gemm_bf16_ws takes for this product (with its workspace): 128, 256 or 512.
MM_API int mm_gemm_tile_rows(int M, int N, int K, int bn) {
    if (M <= 0 || N <= 0 || K <= 0) return 0;
    const int BN = bn == 128 ? 128 : 256;
    return make_plan(M, N, K, BN, sm_count(), BN == 256, true).rows;
}

// Bytes of workspace with which mm_gemm_bf16_ws splits the tail of this product along K (0: it would not).
MM_API long long mm_gemm_ws_bytes(int M, int N, int K, int a_mn, int b_mn, int bn) {
    if (M <= 0 || N <= 0 || K <= 0 || (!a_mn && !b_mn && skinny(M, N, K))) return 0;
    const int BN = bn == 128 ? 128 : 256;
    return split_bytes(make_plan(M, N, K, BN, sm_count(), BN == 256, true), M, N, BN);
}

// lda/ldb/ldc: elements between consecutive rows of the tensors as laid out in memory.
// Requirements: base pointers 16-byte aligned; ld* multiples of 8; `status` is a device int (0 = ok).
// ws: null (the tile list is not split), or workspace of mm_gemm_ws_bytes (16-byte aligned), used by this call alone.
MM_API int mm_gemm_bf16_ws(const void* A, const void* B, void* C, const void* bias, int M, int N, int K, long long lda,
                           long long ldb, long long ldc, int a_mn, int b_mn, int bn, int* status, void* ws, long long ws_bytes,
                           cudaStream_t st) {
    if ((lda | ldb | ldc) % 8) return -1;
    if (((uintptr_t)A | (uintptr_t)B | (uintptr_t)C | (uintptr_t)ws) & 15) return -2;
    if (M <= 0 || N <= 0 || K <= 0) return -3;
    if (!a_mn && !b_mn && skinny(M, N, K)) return mm_gemv_bf16(A, B, bias, nullptr, nullptr, C, M, N, K, lda, ldb, 0, ldc, 0.f, 0, st);
    float* w = (float*)ws;
#define MM_DISPATCH(BN_)                                                                                                              \
    if (!a_mn && !b_mn) return launch<BN_, false, false>(A, B, C, bias, M, N, K, lda, ldb, ldc, status, st, Route(), w, ws_bytes);      \
    if (!a_mn && b_mn) return launch<BN_, false, true>(A, B, C, bias, M, N, K, lda, ldb, ldc, status, st, Route(), w, ws_bytes);        \
    if (a_mn && !b_mn) return launch<BN_, true, false>(A, B, C, bias, M, N, K, lda, ldb, ldc, status, st, Route(), w, ws_bytes);        \
    return launch<BN_, true, true>(A, B, C, bias, M, N, K, lda, ldb, ldc, status, st, Route(), w, ws_bytes);
    if (bn == 128) {
        MM_DISPATCH(128)
    }
    MM_DISPATCH(256)
#undef MM_DISPATCH
}

// Products over the rows in use of a buffer whose number only the device knows: `count` (device int), less `base`, at most M or, with
// a_mn = b_mn = 1, K.
//   NT / NN: C[:count] = op(A)[:count] op(B); rows of C behind them, up to a tile's end, are overwritten.
//   TN:      C = A[:count]^T B[:count]; the operands' rows up to the next multiple of 64 have to be zero.
// ws: workspace of mm_gemm_rows_ws_bytes (16-byte aligned).
MM_API long long mm_gemm_rows_ws_bytes(int M, int N, int K, int a_mn, int b_mn) {
    if (M <= 0 || N <= 0 || K <= 0) return 0;
    const int sms = sm_count();
    const Plan plan = make_plan(M, N, K, 256, sms, true, true, !(a_mn && b_mn));
    if (a_mn && b_mn) return split_bytes(plan, M, N, 256);
    // what the most that any number of rows is cut into takes.  The device is told the room, not the count: its divisions may round otherwise
    const int workers = plan.rows > BM ? sms / 2 : sms;
    int most = 0;
    for (int m = 1; m <= (M + plan.rows - 1) / plan.rows; ++m) {
        const TailPlan t = plan_tail(m * plan.rows, N, K, 256, plan.rows, workers, 16, kMostRounds * workers);
        const int items = t.parts > 1 ? (m * ((N + 255) / 256) - t.full) * t.parts : 0;
        if (items > most) most = items;
    }
    return kPlanBytes + (long long)most * plan.rows * 256 * 4;
}
MM_API int mm_gemm_bf16_rows(const void* A, const void* B, void* C, int M, int N, int K, long long lda, long long ldb, long long ldc, int a_mn,
                             int b_mn, const int* count, int base, int* status, void* ws, long long ws_bytes, cudaStream_t st) {
    if ((lda | ldb | ldc) % 8) return -1;
    if (((uintptr_t)A | (uintptr_t)B | (uintptr_t)C | (uintptr_t)ws) & 15) return -2;
    if (M <= 0 || N <= 0 || K <= 0 || (a_mn && !b_mn)) return -3;
    if (ws_bytes < mm_gemm_rows_ws_bytes(M, N, K, a_mn, b_mn)) return -4;
    Route rt;
    rt.count = count;
    rt.count_base = base;
    rt.counts_depth = a_mn;
    if (a_mn) return launch<256, true, true>(A, B, C, nullptr, M, N, K, lda, ldb, ldc, status, st, rt, (float*)ws, ws_bytes);
    if (b_mn) return launch<256, false, true>(A, B, C, nullptr, M, N, K, lda, ldb, ldc, status, st, rt, (float*)ws, ws_bytes);
    return launch<256, false, false>(A, B, C, nullptr, M, N, K, lda, ldb, ldc, status, st, rt, (float*)ws, ws_bytes);
}

// C[M, F] = silu(A W_gate^T) * (A W_up^T) with W = [W_gate; W_up] stored as one [2F, K] matrix.  F % 128 == 0.
MM_API int mm_gemm_swiglu_bf16(const void* A, const void* W, void* C, int M, int F, int K, long long lda, long long ldw,
                               long long ldc, int* status, cudaStream_t st) {
    if ((lda | ldw | ldc) % 8) return -1;
    if (((uintptr_t)A | (uintptr_t)W | (uintptr_t)C) & 15) return -2;
    if (M <= 0 || F <= 0 || K <= 0 || F % 128) return -3;
    if (skinny(M, 2 * F, K)) return mm_gemv_bf16(A, W, nullptr, nullptr, nullptr, C, M, F, K, lda, ldw, 0, ldc, 0.f, 1, st);
    return launch<256, false, false, true>(A, W, C, nullptr, M, F, K, lda, ldw, ldc, status, st);
}


// Routed output (the collective is the epilogue: slabs are written straight into the destinations' buffers over
// NVLink).  K-major operands (y = x W^T + bias).  mode 1: all-to-all of column blocks (Ulysses head scatter),
// requires blk % 64 == 0; mode 2: push of row blocks into per-source slots (first half of a reduce-scatter),
// requires blk % 128 == 0.  dst[d]: base of destination d's [dst_rows, dst_cols] bf16 buffer with row pitch ldc.
// b_mn = 1: B is stored [K, N] row-major (the NN product of a data-gradient GEMM) instead of [N, K].
MM_API int mm_gemm_bf16_routed_ex(const void* A, const void* B, const void* bias, int M, int N, int K, long long lda,
                                  long long ldb, void* const* dst, long long dst_rows, long long dst_cols, long long ldc,
                                  int mode, int blk, int world, int rank, int row_off, int b_mn, int* status,
                                  cudaStream_t st) {
    if ((lda | ldb | ldc) % 8) return -1;
    if (((uintptr_t)A | (uintptr_t)B) & 15) return -2;
    if (mode == 1 && (blk % 64 || N % (blk * world))) return -3;
    if (mode == 2 && (blk % 128 || M != blk * world)) return -3;
    if (mode != 1 && mode != 2) return -4;
    Route rt;
    rt.mode = mode; rt.blk = blk; rt.world = world; rt.rank = rank; rt.row_off = row_off;
    rt.dst = dst; rt.dst_rows = dst_rows; rt.dst_cols = dst_cols;
    const bool wide = (mode == 1 && blk % 256 == 0) || (mode == 2 && N >= 256);
    if (b_mn) {
        if (wide) return launch<256, false, true>(A, B, nullptr, bias, M, N, K, lda, ldb, ldc, status, st, rt);
        return launch<128, false, true>(A, B, nullptr, bias, M, N, K, lda, ldb, ldc, status, st, rt);
    }
    if (wide) return launch<256, false, false>(A, B, nullptr, bias, M, N, K, lda, ldb, ldc, status, st, rt);
    return launch<128, false, false>(A, B, nullptr, bias, M, N, K, lda, ldb, ldc, status, st, rt);
}

// Mode 1 (K-major operands) with the row statistics side output: stats [M, n_slots] fp32, zeroed by the caller, receives
// the sum of squares of each output row over each of the n_slots equal column groups (q | k | v).
MM_API int mm_gemm_bf16_routed_stats(const void* A, const void* B, const void* bias, int M, int N, int K, long long lda,
                                     long long ldb, void* const* dst, long long dst_rows, long long dst_cols, long long ldc,
                                     int blk, int world, int rank, int row_off, float* stats, int n_slots, int* status,
                                     cudaStream_t st) {
    if ((lda | ldb | ldc) % 8) return -1;
    if (((uintptr_t)A | (uintptr_t)B) & 15) return -2;
    if (blk % 64 || N % (blk * world) || n_slots < 1 || N % n_slots || (N / n_slots) % 64) return -3;
    Route rt;
    rt.mode = 1; rt.blk = blk; rt.world = world; rt.rank = rank; rt.row_off = row_off;
    rt.dst = dst; rt.dst_rows = dst_rows; rt.dst_cols = dst_cols;
    rt.stats = stats; rt.n_slots = n_slots;
    if (blk % 256 == 0) return launch<256, false, false>(A, B, nullptr, bias, M, N, K, lda, ldb, ldc, status, st, rt);
    return launch<128, false, false>(A, B, nullptr, bias, M, N, K, lda, ldb, ldc, status, st, rt);
}

MM_API int mm_gemm_bf16_routed(const void* A, const void* B, const void* bias, int M, int N, int K, long long lda,
                               long long ldb, void* const* dst, long long dst_rows, long long dst_cols, long long ldc,
                               int mode, int blk, int world, int rank, int row_off, int* status, cudaStream_t st) {
    return mm_gemm_bf16_routed_ex(A, B, bias, M, N, K, lda, ldb, dst, dst_rows, dst_cols, ldc, mode, blk, world, rank,
                                  row_off, 0, status, st);
}

// out[r, :] = sum_s slots[s * rows + r, :]   (second half of the reduce-scatter: fold the per-source slots)
namespace {
__global__ void fold_slots_kernel(const bf16* __restrict__ slots, bf16* __restrict__ out, long long rows, int cols,
                                  long long pitch, int world) {
    let_successor_start();
    const int cv = cols >> 3;
    const long long total = rows * cv;
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (long long)gridDim.x * blockDim.x) {
        const long long r = i / cv;
        const int c = (int)(i - r * cv);
        float acc[8] = {0, 0, 0, 0, 0, 0, 0, 0};
        for (int s = 0; s < world; ++s) {
            float f[8];
            unpack8(reinterpret_cast<const Vec8*>(slots + (s * rows + r) * pitch)[c], f);
#pragma unroll
            for (int k = 0; k < 8; ++k) acc[k] += f[k];
        }
        reinterpret_cast<Vec8*>(out + r * cols)[c] = pack8(acc);
    }
}
}  // namespace

MM_API int mm_fold_slots(const void* slots, void* out, long long rows, int cols, long long pitch, int world, cudaStream_t st) {
    if (cols % 8 || pitch % 8) return -1;
    long long work = rows * (cols / 8);
    int grid = (int)((work + 255) / 256 < 148 * 8 ? (work + 255) / 256 : 148 * 8);
    fold_slots_kernel<<<grid < 1 ? 1 : grid, 256, 0, st>>>((const bf16*)slots, (bf16*)out, rows, cols, pitch, world);
    return (int)cudaGetLastError();
}
