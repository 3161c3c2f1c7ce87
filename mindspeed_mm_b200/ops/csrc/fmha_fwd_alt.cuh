// Forward flash-attention kernel with alternating softmax groups.  Included by fmha_fwd.cu inside its namespace.
//
// One CTA = one 128-row query tile of one head:
//   warp 0      TMA producer: K_j, V_j (rings of 3)
//   warp 1      issues S_j = Q K_j^T, as soon as the softmax has taken S_{j-2} into registers
//   warps 4-7   softmax of the even key tiles, warps 8-11 of the odd ones: thread = query row, all 128 columns of S in registers;
//               writes P (bf16 pairs) to its own place in tensor memory, the A operand of PV
//   warp 2      issues O += P_j V_j
// TMEM: S_even | S_odd | O (128 columns each) | Q | P (64 columns of bf16 pairs each).  Q is an A operand from tensor memory because
// a 128 x 128 x 16 product that takes A from shared memory runs at about half rate (130 - 150 clocks against 72).  P does not lie
// over S, and each product has an issuing warp of its own, so that neither the next scores nor their 100 clocks per wait and
// commit stand in the chain of a tile: the two groups work through their tiles back to back, one tile apart, and only P waits for
// the PV product before it.  What has to go from tile to tile is the row's reference maximum, which a group hands to the other one
// through shared memory as soon as it knows it, before its exponentials.
// O is accumulated in tensor memory with lazy rescaling: the reference moves only when the running maximum has grown by more than
// 2^8 since it was set, and then the row's thread rescales its O columns (after PV of the tile before, ahead of its own P).
// P = exp2(S * scale - m_ref) is at most 2^8, and l, the LSE and O refer to the same m_ref, so the result is exact.
// Bound by the length of a group's loop (3300 clocks for its tile: 1340 of them exponentials at the special-function rate, the
// rest the latencies of tensor-memory reads and of five barrier waits), and next by P, whose one buffer takes 1300 clocks a tile.
// 40 heads of 32760 x 32760, head dim 128: 20.2 ms, 1090 TFLOP/s (one group with P over S: 24.3 ms).

constexpr int kAltThreads = 3 * 128;
// Registers: 168 a thread at launch (12 warps); the warpgroup of producer and issuers gives its share to the two softmax groups,
// which hold a row of 128 scores each.  40 + 2 * 232 = 3 * 168.
constexpr int kAltRegsLow = 40, kAltRegsHigh = 232;
static_assert(kAltRegsLow + 2 * kAltRegsHigh <= 3 * 168, "register shares of the launch");
constexpr int kAltK = 3, kAltV = 3;
constexpr int kAltSmem = (kAltK + kAltV) * kTileBytes + 256 + 4 * 128 * 4 + 1024;    // + barriers + m, l of both groups + alignment

__global__ void __launch_bounds__(kAltThreads, 1)
fmha_fwd_alt_kernel(const __grid_constant__ CUtensorMap tmK, const __grid_constant__ CUtensorMap tmV, FmhaParams p) {
    wait_for_predecessor();
    if ((int)tile_of(p.heads_first) >= *p.n_tiles) return;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint8_t* sK = smem;
    uint8_t* sV = sK + kAltK * kTileBytes;
    uint64_t* bars = reinterpret_cast<uint64_t*>(sV + kAltV * kTileBytes);
    uint64_t* q_full = bars + 0;
    uint64_t* k_full = bars + 1;                         // [3]
    uint64_t* k_empty = bars + 4;                        // [3]
    uint64_t* v_full = bars + 7;                         // [3]
    uint64_t* v_empty = bars + 10;                       // [3]  PV(j) complete: V's stage and P are free, O is up to date
    uint64_t* s_full = bars + 13;                        // [2]
    uint64_t* s_free = bars + 15;                        // [2]  S is in registers
    uint64_t* p_full = bars + 17;
    uint64_t* m_ready = bars + 18;                       // [2][4 row quarters]
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 26);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
    float* m_ref = reinterpret_cast<float*>(reinterpret_cast<uint8_t*>(bars) + 256);      // [group][128]
    float* l_part = m_ref + 2 * 128;                                                      // [group][128]

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int seq = p.tile_seq[tile_of(p.heads_first)], q0 = p.tile_q0[tile_of(p.heads_first)], nseq = p.tile_nseq[tile_of(p.heads_first)];
    const int head = head_of(p.heads_first), kv_head = head / (p.Nq / p.Nkv);
    const int q_begin = p.cu_q[seq], q_len = p.cu_q[seq + nseq] - q_begin;
    const int k_begin = p.cu_k[seq], k_len = p.cu_k[seq + nseq] - k_begin;
    const int diag = k_len - q_len;                      // causal: key j visible to query i iff j <= i + diag
    const int kv_end = p.causal ? min(k_len, q0 + BQ + diag) : k_len;
    const int n_kv = kv_end > 0 ? (kv_end + BKV - 1) / BKV : 0;

    if (threadIdx.x == 0) {
        mbar_init(q_full, 256);
        mbar_init(p_full, 4);                            // one arrival per warp
        for (int i = 0; i < 2; ++i) {
            mbar_init(&s_full[i], 1);
            mbar_init(&s_free[i], 4);
        }
        for (int i = 0; i < 3; ++i) {
            mbar_init(&k_full[i], 1);
            mbar_init(&k_empty[i], 1);
            mbar_init(&v_full[i], 1);
            mbar_init(&v_empty[i], 1);
        }
        for (int i = 0; i < 8; ++i) mbar_init(&m_ready[i], 1);
        *abort_flag = 0;
        fence_barrier_init();
        prefetch_tmap(&tmK);
        prefetch_tmap(&tmV);
    }
    if (warp == 1) {
        tmem_alloc(tmem_slot, 512);
        tmem_relinquish();
    }
    fence_before_sync();
    __syncthreads();
    fence_after_sync();
    const uint32_t tmem_base = *tmem_slot;
    let_successor_start();           // behind the allocation, see common.cuh
    const uint32_t tS = tmem_base, tO = tmem_base + 256, tQ = tmem_base + 384, tP = tmem_base + 448;

    if (warp < 4) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kAltRegsLow));
    if (warp == 0) {
        // ------------------------------------------------------------------------------ TMA producer
        if (lane == 0) {
            for (int j = 0; j < n_kv; ++j) {
                const int ks = j % kAltK, vs = j % kAltV, row = k_begin + j * BKV;
                if (!mbar_wait(&k_empty[ks], ((j / kAltK) & 1) ^ 1, abort_flag)) { atomicExch(p.status, MM_TIMEOUT_TMA); break; }
                mbar_expect_tx(&k_full[ks], kTileBytes);
                tma_load_3d(sK + ks * kTileBytes, &tmK, &k_full[ks], 0, kv_head, row);
                tma_load_3d(sK + ks * kTileBytes + kAtomBytes, &tmK, &k_full[ks], 64, kv_head, row);
                if (!mbar_wait(&v_empty[vs], ((j / kAltV) & 1) ^ 1, abort_flag)) { atomicExch(p.status, MM_TIMEOUT_TMA); break; }
                mbar_expect_tx(&v_full[vs], kTileBytes);
                tma_load_3d(sV + vs * kTileBytes, &tmV, &v_full[vs], 0, kv_head, row);
                tma_load_3d(sV + vs * kTileBytes + kAtomBytes, &tmV, &v_full[vs], 64, kv_head, row);
            }
        }
    } else if (warp == 1) {
        // ------------------------------------------------------------------------------ scores
        if (lane == 0 && n_kv > 0) {
            constexpr uint32_t idesc_qk = idesc_bf16(BQ, BKV, 0, 0);
            const int dsteps = (p.D + 15) / 16;          // a narrow head's zero columns are left out of both products
            bool ok = mbar_wait(q_full, 0, abort_flag);
            for (int j = 0; j < n_kv && ok; ++j) {
                const int st = j & 1, ks = j % kAltK;
                ok = mbar_wait(&k_full[ks], (j / kAltK) & 1, abort_flag) && mbar_wait(&s_free[st], ((j >> 1) & 1) ^ 1, abort_flag);
                if (!ok) break;
                fence_after_sync();
                const uint32_t ka = smem_u32(sK + ks * kTileBytes);
#pragma unroll
                for (int k = 0; k < HD / 16; ++k)
                    if (k < dsteps)
                        mma_ts(tS + st * 128, tQ + k * 8, smem_desc_sw128(ka + (k >> 2) * kAtomBytes + (k & 3) * 32, 16, 1024), idesc_qk,
                               k ? 1u : 0u);
                mma_commit(&s_full[st]);
                mma_commit(&k_empty[ks]);
            }
            if (!ok) atomicExch(p.status, MM_TIMEOUT_MMA);
        }
    } else if (warp == 2) {
        // ------------------------------------------------------------------------------ values
        if (lane == 0) {
            const uint32_t idesc_pv = idesc_bf16(BQ, (p.D + 15) / 16 * 16, 0, 1);
            bool ok = true;
            for (int j = 0; j < n_kv && ok; ++j) {
                const int vs = j % kAltV;
                ok = mbar_wait(&v_full[vs], (j / kAltV) & 1, abort_flag) && mbar_wait(p_full, j & 1, abort_flag);
                if (!ok) break;
                fence_after_sync();
                const uint32_t va = smem_u32(sV + vs * kTileBytes);
#pragma unroll
                for (int k = 0; k < BKV / 16; ++k)
                    mma_ts(tO, tP + k * 8, smem_desc_sw128(va + k * 2048, kAtomBytes, 1024), idesc_pv, (j | k) ? 1u : 0u);
                mma_commit(&v_empty[vs]);
            }
            if (!ok) atomicExch(p.status, MM_TIMEOUT_MMA);
        }
    }
    } else {
        asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kAltRegsHigh));
        // ------------------------------------------------------------------------------ softmax (warps 4..11)
        const int grp = (warp - 4) >> 2;                 // key tiles j = grp, grp + 2, ..
        const int qd = warp & 3;                         // TMEM lane quarter this warp may touch
        const int row = qd * 32 + lane, qi = q0 + row;
        const uint32_t lane_off = (uint32_t)(qd * 32) << 16, t_s = tS + grp * 128 + lane_off, t_o = tO + lane_off, t_p = tP + lane_off;
        int vis_lo = 0, vis_hi = k_len;                  // keys this row may see (packed tiles: its own sequence)
        if (nseq > 1) packed_row_range(p.cu_q, seq, nseq, q_begin + qi, q_begin, vis_lo, vis_hi);
        if (n_kv > 0) {                                  // half a row of Q per thread -> tensor memory
            const bf16* src = p.q + (size_t)(q_begin + qi) * p.q_ts + (size_t)head * p.D + grp * 64;
            uint32_t r[32];
#pragma unroll
            for (int g = 0; g < 8; ++g) {
                const uint4 v = qi < q_len && grp * 64 + g * 8 < p.D ? reinterpret_cast<const uint4*>(src)[g] : make_uint4(0, 0, 0, 0);
                r[4 * g] = v.x;
                r[4 * g + 1] = v.y;
                r[4 * g + 2] = v.z;
                r[4 * g + 3] = v.w;
            }
            tmem_st_32x32(tQ + grp * 32 + lane_off, r);
            tmem_wait_st();
            fence_before_sync();
            mbar_arrive(q_full);
        }
        float m = -INFINITY, l = 0.f;                    // reference of this group's last tile, and its row sum
        bool ok = true;
        for (int j = grp; j < n_kv; j += 2) {
            // (the votes keep the warp together: the tensor-memory accesses below are whole-warp instructions)
            if (!__all_sync(0xffffffffu, mbar_wait(&s_full[grp], (j >> 1) & 1, abort_flag))) { ok = false; break; }
            fence_after_sync();
            uint32_t r[128];
#pragma unroll
            for (int c = 0; c < 4; ++c) tmem_ld_32x32(t_s + c * 32, r + c * 32);
            float m_prev = -INFINITY;                     // reference after tile j - 1; fetched while the scores are on their way
            if (j > 0) {
                if (!__all_sync(0xffffffffu, mbar_wait(&m_ready[(grp ^ 1) * 4 + qd], ((j - 1) >> 1) & 1, abort_flag))) { ok = false; break; }
                m_prev = m_ref[(grp ^ 1) * 128 + row];
            }
            tmem_wait_ld();
            fence_before_sync();
            __syncwarp();
            if (lane == 0) mbar_arrive(&s_free[grp]);
            const int kbase = j * BKV;
            if (kbase + BKV > k_len || (p.causal && kbase + BKV - 1 > q0 + diag) || nseq > 1) {
                const int hi = (p.causal ? min(k_len - 1, qi + diag) : vis_hi - 1) - kbase, lo = vis_lo - kbase;
#pragma unroll
                for (int i = 0; i < 128; ++i)
                    if (i > hi || i < lo) r[i] = 0xff800000u;                                       // -inf
            }
            float mx[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
            for (int i = 0; i < 128; i += 8)              // four chains of three-input maxima over the raw scores (scale > 0)
#pragma unroll
                for (int c = 0; c < 4; ++c) mx[c] = max3(mx[c], __uint_as_float(r[i + 2 * c]), __uint_as_float(r[i + 2 * c + 1]));
            const float mx_all = fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3])) * p.scale_log2;
            const bool grow = mx_all > m_prev + 8.f;      // also true for the first finite maximum (m_prev = -inf)
            const float m_new = grow ? mx_all : m_prev;
            m_ref[grp * 128 + row] = m_new;
            __syncwarp();
            if (lane == 0) mbar_arrive(&m_ready[grp * 4 + qd]);
            const float m_use = m_new == -INFINITY ? 0.f : m_new;
            l *= exp2f(m - m_use);                        // m = -inf before the first tile -> 0; 1 while the reference stays
            m = m_new;
            const float2 sc2 = make_float2(p.scale_log2, p.scale_log2), ng2 = make_float2(-m_use, -m_use);
            float2 sum_a = make_float2(0.f, 0.f), sum_b = make_float2(0.f, 0.f);
#pragma unroll
            for (int i = 0; i < 64; i += 2) {             // two packed chains: exp2(s * scale - m), running sums, bf16 pairs
                const float2 x0 = __ffma2_rn(make_float2(__uint_as_float(r[2 * i]), __uint_as_float(r[2 * i + 1])), sc2, ng2);
                const float2 x1 = __ffma2_rn(make_float2(__uint_as_float(r[2 * i + 2]), __uint_as_float(r[2 * i + 3])), sc2, ng2);
                const float2 e0 = make_float2(exp2f(x0.x), exp2f(x0.y)), e1 = make_float2(exp2f(x1.x), exp2f(x1.y));
                sum_a = __fadd2_rn(sum_a, e0);
                sum_b = __fadd2_rn(sum_b, e1);
                bf162 t0 = __floats2bfloat162_rn(e0.x, e0.y), t1 = __floats2bfloat162_rn(e1.x, e1.y);
                r[i] = *reinterpret_cast<uint32_t*>(&t0);
                r[i + 1] = *reinterpret_cast<uint32_t*>(&t1);
            }
            if (j > 0) {                                  // P(j - 1) has been used, O holds the tiles before this one
                if (!__all_sync(0xffffffffu, mbar_wait(&v_empty[(j - 1) % kAltV], ((j - 1) / kAltV) & 1, abort_flag))) { ok = false; break; }
                fence_after_sync();
                if (__any_sync(0xffffffffu, grow)) {
                    const float a = grow ? exp2f(m_prev - m_use) : 1.f;
                    const float2 a2 = make_float2(a, a);
#pragma unroll 1
                    for (int c = 0; c < 128; c += 16) {
                        if (c >= p.D) break;
                        uint32_t o[16];
                        tmem_ld_32x16(t_o + c, o);
                        tmem_wait_ld();
#pragma unroll
                        for (int i = 0; i < 8; ++i) {
                            const float2 v = __fmul2_rn(make_float2(__uint_as_float(o[2 * i]), __uint_as_float(o[2 * i + 1])), a2);
                            o[2 * i] = __float_as_uint(v.x);
                            o[2 * i + 1] = __float_as_uint(v.y);
                        }
                        tmem_st_32x16(t_o + c, o);
                    }
                }
            }
            tmem_st_32x32(t_p, r);
            tmem_st_32x32(t_p + 32, r + 32);
            l += (sum_a.x + sum_a.y) + (sum_b.x + sum_b.y);
            tmem_wait_st();
            fence_before_sync();
            __syncwarp();
            if (lane == 0) mbar_arrive(p_full);
        }
        if (n_kv > 0) {
            if (ok) ok = __all_sync(0xffffffffu, mbar_wait(&v_empty[(n_kv - 1) % kAltV], ((n_kv - 1) / kAltV) & 1, abort_flag));
            l_part[grp * 128 + row] = l;
            if (grp < n_kv) m_ref[grp * 128 + row] = m;
            else m_ref[grp * 128 + row] = -INFINITY;     // a single key tile: the odd group had none
        }
        named_barrier_sync(1, 256);                      // a warp whose wait gave up still takes part
        if (n_kv > 0 && ok) {
            fence_after_sync();
            // the group of the last tile knows the final reference; the other group's sum refers to its own last one
            const int g_last = (n_kv - 1) & 1;
            const float m_fin = m_ref[g_last * 128 + row], m_use = m_fin == -INFINITY ? 0.f : m_fin;
            const float lsum = l_part[g_last * 128 + row] + l_part[(g_last ^ 1) * 128 + row] * exp2f(m_ref[(g_last ^ 1) * 128 + row] - m_use);
            const float inv = lsum > 0.f ? 1.f / lsum : 0.f;
            bf16* dst = p.o + ((size_t)(q_begin + qi) * p.Nq + head) * p.D + grp * 64;
#pragma unroll 1
            for (int c = 0; c < 64; c += 16) {            // a group stores half of the columns
                if (grp * 64 + c >= p.D) break;
                uint32_t o[16];
                tmem_ld_32x16(t_o + grp * 64 + c, o);
                tmem_wait_ld();
#pragma unroll
                for (int g = 0; g < 2; ++g) {
                    float f[8];
#pragma unroll
                    for (int i = 0; i < 8; ++i) f[i] = __uint_as_float(o[g * 8 + i]) * inv;
                    if (qi < q_len && grp * 64 + c + g * 8 < p.D) reinterpret_cast<Vec8*>(dst)[c / 8 + g] = pack8(f);
                }
                __syncwarp();
            }
            if (grp == 0 && qi < q_len)
                p.lse[(size_t)head * p.T + q_begin + qi] = (m_fin == -INFINITY) ? -INFINITY : m_fin * 0.6931471805599453f + logf(lsum);
        }
        if (n_kv == 0 && qi < q_len) {                   // no key is visible to this tile
            bf16* dst = p.o + ((size_t)(q_begin + qi) * p.Nq + head) * p.D + grp * 64;
            for (int g = 0; g < 8; ++g)
                if (grp * 64 + g * 8 < p.D) reinterpret_cast<uint4*>(dst)[g] = make_uint4(0, 0, 0, 0);
            if (grp == 0) p.lse[(size_t)head * p.T + q_begin + qi] = -INFINITY;
        }
        if (!ok && lane == 0) atomicExch(p.status, MM_TIMEOUT_EPI);
    }

    if (*abort_flag)
        for (int i = 0; i < 64; ++i) __nanosleep(1000);
    fence_before_sync();
    __syncthreads();
    if (warp == 1) {
        fence_after_sync();
        tmem_dealloc(tmem_base, 512);
    }
}
