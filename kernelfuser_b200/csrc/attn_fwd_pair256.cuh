// Persistent, warp-specialised tcgen05 flash-attention forward kernel for head dim 256 on SM PAIRS.
//
// Same operator, pipeline and roles as attn_fwd_persist256.cuh (reference: `attention_v2_kernel`,
// src/e1_rope_publication_v1.py:609-649), for models whose query heads share KV heads in even numbers.  A cluster of
// two CTAs works on two query heads of one KV head at the same query block (identical causal bounds), each CTA on
// its own 128-row tile with its own softmax, Q and epilogue warps; the MMAs are tcgen05.mma.cta_group::2 of 256
// rows, issued by CTA 0 for both, whose B operand (K or V) is split between the two shared memories.
//
// What bounds it: at this head dim a CTA of its own streams 64 KB of K and V per 64-key sub-block for 128 query rows, and
// 148 of them pull that from L2 together (~1550 clocks per sub-block where the MMAs take 1024).  A pair copies every K/V
// tile once for 256 rows - each CTA loads 32 of the 64 keys of K and half of the columns of V - so the stream halves,
// and the ring holds five sub-blocks instead of two and a half.  What is left is the chain P V, Q K^T, hand-over,
// softmax of a score buffer (~1400 clocks per sub-block with everything that a tile adds); large launches run at the
// 1 kW power limit.  B200, one CTA per tile -> pairs, each by itself back to back: B=8 S=8192 16/8 heads 3917 -> 3556 us;
// in blocks of 30 ms, its 8-GPU shard 502 -> 459, B=1 S=16384 4/2 heads 473 -> 426.
//
// Barriers.  What the issuer waits for lives in CTA 0; what it signals - tcgen05.commit with both CTAs' mask - arrives at
// the same offset in both.  A K/V stage is full when the halves of both CTAs have landed: each CTA announces its half
// on CTA 0's barrier and its TMA copy (.cta_group::2, into its own shared memory) completes there, so the barrier that the
// issuer waits on is that of the copies themselves.  (With a relay in CTA 1 that waits for its copy and tells CTA 0
// in a release that CTA 0 acquires at cluster scope, B=8 S=8192 16/8 heads took 4843 us against 3556; under ncu B=2
// S=4096 takes 397 k cycles, 407 k with a relay that orders nothing.)  Tensor memory is handed over with relaxed arrivals:
// tcgen05.wait and tcgen05.fence order its accesses.  Work items are claimed by CTA 0's scheduler and published to both
// CTAs.
#pragma once
#include "attn_fwd_persist256.cuh"

namespace kf {

constexpr int kPrRing = 10;                             // K/V ring stages: half a 64-key tile of K or V each
constexpr int kPrStageBytes = kSub * 128 * 2;           // K: 32 keys x 256 columns; V: 64 keys x 128 columns (16 KB)
constexpr int kPrKBoxBytes = (kSub / 2) * 128;          // 32 rows x 64 columns
constexpr int kPrVBoxBytes = kSub * 128;                // 64 rows x 64 columns
// Published work items in flight.  No role trails the claim of a new item by more than three items (an epilogue still
// running holds back the next item's first P V, and with it the claim after that), so a slot is free when it is
// written again.
constexpr int kPrItemRing = 8;
constexpr int kPrSmemBytes = kP2QBytes + kPrRing * kPrStageBytes + 1024 + kPsCtrlBytes;
static_assert(kPrSmemBytes <= 232448, "shared memory of an SM");

// Pair item `idx` in the order of sg_decode; `rank` picks the head.
__device__ __forceinline__ P2Item pr_decode(int idx, uint32_t rank, const AttnArgs& a) {
    P2Item it;
    const int G = a.Hq / a.Hkv, pairs = G / 2;
    const int n_mblk = (a.S + kBM - 1) / kBM;
    const int n_sub_all = (a.S + kSub - 1) / kSub;
    const SgItem sg = sg_decode(idx, a.B * a.Hkv, a.sg_groups, a.sg_first, n_mblk, pairs);
    it.b = sg.grp / a.Hkv;
    it.kh = sg.grp % a.Hkv;
    it.m0 = (n_mblk - 1 - sg.level) * kBM;
    it.h = it.kh * G + 2 * sg.sub + static_cast<int>(rank);
    it.nsub = a.causal ? min((it.m0 + kBM) / kSub, n_sub_all) : n_sub_all;
    return it;
}

struct PrCtrl {
    // waited for by CTA 0's issuer: arrivals of both CTAs
    uint64_t q_ready;            // 8 Q-group warps: the tile's prepared Q is in TMEM
    uint64_t o_free;             // 8 Q-group warps: the finished tile's output has been read
    uint64_t p_ready[2];         // [buffer] 8 softmax warps
    uint64_t kv_full[kPrRing];   // both CTAs' halves (1 arrival + bytes each)
    // signalled by the issuer's commits, in both CTAs
    uint64_t kv_empty[kPrRing];
    uint64_t s_full[2];          // [buffer]
    uint64_t pv_done[2];         // [g & 1]
    uint64_t qk_done;            // every Q K^T of the tile has completed (the Q columns may be overwritten)
    uint64_t mma_done;           // every MMA of the launch has completed
    // within a CTA
    uint64_t q_full;             // raw Q of the next tile is in the Q buffer
    uint64_t q_free;             // Q group (4): the Q buffer has been copied out and may be refilled
    uint64_t den_full;           // softmax (4) -> Q group
    uint64_t den_free;           // Q group (4) -> softmax
    uint64_t item_full[kPrItemRing];
    uint64_t near_end;           // CTA 0: softmax -> scheduler
    uint32_t tmem_slot;
    int abort_flag;
    int item[kPrItemRing];
    int dead;
    int issued[2];               // CTA 0: K/V copies that each CTA has issued
    float den[kBM];
};
static_assert(sizeof(PrCtrl) <= kPsCtrlBytes, "control block too large");

// Bounded, abortable wait that also sees what the other CTA released.
__device__ __forceinline__ bool pr_wait(uint64_t* bar, uint32_t parity, volatile int* abort_flag) {
    if (mbar_try_wait_cluster(bar, parity)) return true;
    const long long t0 = clock64();
    uint32_t spins = 0;
    while (true) {
        if (mbar_try_wait_cluster(bar, parity)) return true;
        if ((++spins & 31u) == 0) {
            if (*abort_flag != 0) return false;
            if (clock64() - t0 > kWaitCycles) return false;
        }
    }
}

__device__ __forceinline__ int pr_take_item(PrCtrl* c, int n, int& fail) {
    const int s = n & (kPrItemRing - 1);
    if (!pr_wait(c->item_full + s, (n / kPrItemRing) & 1, &c->abort_flag)) {
        fail = kStatusP2Item;
        return -1;
    }
    return *reinterpret_cast<volatile int*>(c->item + s);
}

template <typename T>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kP2Threads, 1)
attn_fwd_pair256_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_k,
                           const __grid_constant__ CUtensorMap tm_v, const AttnArgs a, const int n_items) {
    constexpr int D = 256;
    constexpr int NB = D / 64;
    constexpr uint32_t kTmemCols = 512;
    constexpr uint32_t kColO = 128, kColQ = 384;
    constexpr uint32_t kIdescQK = umma_idesc(Num<T>::kFmt, 0, 2 * kBM, kSub);
    constexpr uint32_t kIdescPV = umma_idesc(Num<T>::kFmt, 1, 2 * kBM, D);

    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint8_t* smem_q = smem;                       // 128 rows x 256 columns
    uint8_t* smem_kv = smem + kP2QBytes;          // [stage] 16 KB each
    PrCtrl* c = reinterpret_cast<PrCtrl*>(smem_kv + kPrRing * kPrStageBytes);
    volatile int* s_abort = &c->abort_flag;
    const uint32_t rank = cluster_ctarank();
    const bool leader = rank == 0;

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;

    if (tid == 0) {
        prefetch_tensormap(&tm_q);
        prefetch_tensormap(&tm_k);
        prefetch_tensormap(&tm_v);
        mbar_init(&c->q_full, 1);
        mbar_init(&c->q_ready, 8);
        mbar_init(&c->q_free, 4);
        mbar_init(&c->qk_done, 1);
        mbar_init(&c->mma_done, 1);
        mbar_init(&c->o_free, 8);
        mbar_init(&c->den_full, 4);
        mbar_init(&c->den_free, 4);
        mbar_init(&c->near_end, 1);
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            mbar_init(c->s_full + i, 1);
            mbar_init(c->p_ready + i, 8);
            mbar_init(c->pv_done + i, 1);
        }
#pragma unroll
        for (int i = 0; i < kPrRing; ++i) {
            mbar_init(c->kv_full + i, 2);
            mbar_init(c->kv_empty + i, 1);
        }
#pragma unroll
        for (int i = 0; i < kPrItemRing; ++i) mbar_init(c->item_full + i, 1);
        c->abort_flag = 0;
        // an earlier launch or CTA failed: every thread of the pair takes the same decision from CTA 0's copy
        c->dead = *reinterpret_cast<volatile int*>(a.status);
        fence_mbar_init();
    }
    if (warp == 0) {
        __syncwarp();
        tmem_alloc_pair(&c->tmem_slot, kTmemCols);
        tmem_relinquish_pair();
    }
    tc_fence_before();
    __syncthreads();
    cluster_sync();  // barriers of both CTAs are initialised, both have their TMEM
    tc_fence_after();
    const uint32_t tmem_base = c->tmem_slot;
    const bool dead = remote_load(map_to_cta(&c->dead, 0)) != 0;
    // a role that fails records its code and stops both CTAs
    auto give_up = [&](int code) {
        *s_abort = 1;
        remote_store(map_to_cta(&c->abort_flag, rank ^ 1u), 1);
        atomicCAS(a.status, 0, code);
    };

    // Last step of the issuer and of CTA 1's producer: the asynchronous MMAs and the arrivals of their commits end before either CTA frees
    // its TMEM or leaves.  `tiles` ring stages of `items` items have been consumed; a launch that gives up waits for
    // the MMAs that were issued only.  (Every wait is bounded.)
    auto drain_mma = [&](int items, int tiles, bool failed) {
        mbar_wait(&c->mma_done, 0);
        if (failed) return;
        for (int i = 0; i < kPrRing; ++i)
            if (tiles > i) mbar_wait_abortable(c->kv_empty + i, ((tiles - 1 - i) / kPrRing) & 1, s_abort);
        const int last = tiles / 2 - 1;  // last sub-block
        mbar_wait_abortable(c->pv_done + (last & 1), (last >> 1) & 1, s_abort);
        if (last > 0) mbar_wait_abortable(c->pv_done + ((last - 1) & 1), ((last - 1) >> 1) & 1, s_abort);
        mbar_wait_abortable(&c->qk_done, (items - 1) & 1, s_abort);
    };

    int fail = 0;
    int kv_issued = 0, q_issued = 0;  // bookkeeping of the two producers for the exit path

    if (dead) {
        // nothing to do: fall through to the common exit
    } else if (warp < 4) {
        asm volatile("setmaxnreg.inc.sync.aligned.u32 208;");
        // ============================================ softmax
        const int r = tid;
        const uint32_t lane_base = tmem_base + (static_cast<uint32_t>(warp * 32) << 16);
        const float cs = a.scale_log2e;
        const uint32_t p_ready0 = map_to_cta(c->p_ready, 0);
        int g = 0;  // sub-blocks processed so far (all tiles)
        for (int n = 0; !fail; ++n) {
            const int idx = pr_take_item(c, n, fail);
            if (idx < 0) break;
            const P2Item it = pr_decode(idx, rank, a);
            const int row = it.m0 + r;
            RowSoftmax rs;
            for (int jj = 0; jj < it.nsub; ++jj) {
                const int gg = g + jj;
                const int buf = gg & 1;
                const int n0 = jj * kSub;
                const uint32_t col_sb = buf * kSub;
                // tell the scheduler when this tile has only a few sub-blocks left: only then does it claim the next
                if (leader && tid == 0 && jj == max(0, it.nsub - kP2ClaimAhead)) mbar_arrive(&c->near_end);
                if (!mbar_wait_abortable(c->s_full + buf, (gg >> 1) & 1, s_abort)) { fail = kStatusP2SFull; break; }
                tc_fence_after();
                const bool plain = jj > 0 && n0 + kSub <= a.S && (!a.causal || n0 + kSub - 1 <= it.m0);
                if (!plain || !softmax_ordinary<T, kPolyPairsOneTile, false>(lane_base + col_sb, cs, rs)) {
                    const int lim = (a.causal ? min(row + 1, a.S) : a.S) - n0;  // keys of this sub-block that the row sees
                    rs = softmax_general<D, T, kPolyPairsOneTile>(
                        lane_base + col_sb, lane_base + kColO, cs, lim, rs,
                        jj > 0 ? c->pv_done + ((gg - 1) & 1) : nullptr, ((gg - 1) >> 1) & 1, s_abort);
                    if (!rs.ok) { fail = kStatusP2PvDone; break; }
                }
                tmem_wait_st();
                tc_fence_before();
                __syncwarp();
                if (lane == 0) remote_arrive_relaxed(p_ready0 + 8 * buf);
            }
            if (fail) break;
            g += it.nsub;
            // Hand the row sums to the epilogue group.  One buffer: wait until it has read the previous tile's
            // (it signals den_free after reading them); a tile of one or two sub-blocks can get here before any of
            // its P V has been issued, so this wait is not implied by the pipeline.
            if (n > 0 && !mbar_wait_abortable(&c->den_free, (n - 1) & 1, s_abort)) { fail = kStatusP2OFree; break; }
            c->den[r] = rs.den;
            __syncwarp();
            if (lane == 0) mbar_arrive(&c->den_full);
        }
        if (fail) give_up(fail);
    }
    else if (warp < 8) {
        // ============================================ Q transform, Q -> TMEM, output epilogue (keeps its 168 registers)
        const int r = tid - 128;                       // 0..127: row of the tile, TMEM lane
        const uint32_t lane_base = tmem_base + (static_cast<uint32_t>((warp & 3) * 32) << 16);
        int gsub = 0;                                  // sub-blocks of the tiles whose epilogue has been done
        // next tile: wait for its raw Q, transform it in place (RMSNorm + gamma + RoPE); returns its index or -1
        auto prepare_next = [&](int n) -> int {
            const int idx = pr_take_item(c, n, fail);
            if (idx < 0) return -1;
            const P2Item it = pr_decode(idx, rank, a);
            bool waited = false, ok = true;
            auto wait_q = [&]() {
                if (waited) return ok;
                waited = true;
                // (all lanes of a warp wait here together; the vote keeps them together if the wait runs out)
                ok = __all_sync(0xffffffffu, mbar_wait_abortable(&c->q_full, n & 1, s_abort)) != 0;
                return ok;
            };
            if (a.fuse_q) q_prologue_coop<D, T, 4>(smem_q, r, it.m0, a, wait_q);
            if (!wait_q()) { fail = kStatusP2QFull; return -1; }
            return idx;
        };
        // the prepared Q moves from shared memory into TMEM columns [kColQ, kColQ + 128): thread r copies row r
        auto q_to_tmem = [&](int n) {
            // every row has been transformed by some thread of this group: make that visible to the copier
            // (the barrier also makes the outcome of the waits uniform across the group)
            if (named_barrier_or(2, 128, fail != 0)) { if (!fail) fail = kStatusP2QFull; return; }
            const uint8_t* qrow = smem_q + r * 128;
            const int sw = r & 7;
#pragma unroll
            for (int bx = 0; bx < NB; ++bx) {
                uint32_t w[32];
#pragma unroll
                for (int ch = 0; ch < 8; ++ch) {
                    const uint4 u = *reinterpret_cast<const uint4*>(qrow + bx * kBoxBytes + ((ch ^ sw) << 4));
                    w[ch * 4 + 0] = u.x; w[ch * 4 + 1] = u.y; w[ch * 4 + 2] = u.z; w[ch * 4 + 3] = u.w;
                }
                tmem_st32(lane_base + kColQ + bx * 32, w);
            }
            tmem_wait_st();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) {
                remote_arrive_relaxed(map_to_cta(&c->q_ready, 0));
                mbar_arrive(&c->q_free);
            }
            (void)n;
        };
        // (Waits are per thread and bounded; before the group meets at a barrier, a vote makes their outcome
        // uniform, so a wait that ran out in some threads cannot leave the others stuck at that barrier.)
        auto group_failed = [&]() {
            if (named_barrier_or(3, 128, fail != 0)) {
                if (!fail) fail = kStatusP2QFull;
                return true;
            }
            return false;
        };
        int cur = prepare_next(0);
        if (!group_failed() && cur >= 0) q_to_tmem(0);
        for (int n = 0; cur >= 0 && !fail; ++n) {
            const P2Item it = pr_decode(cur, rank, a);
            // ---- next tile: transform its Q while this one computes, move it into TMEM once this tile's last
            // Q K^T has completed (the tile then still has a sub-block of softmax and P V to go)
            const int nxt = prepare_next(n + 1);
            if (group_failed()) break;
            if (nxt >= 0) {
                if (!mbar_wait_abortable(&c->qk_done, n & 1, s_abort)) fail = kStatusP2QkDone;
                tc_fence_after();
                q_to_tmem(n + 1);  // (its barrier makes `fail` uniform)
                if (fail) break;
            }
            // ---- epilogue of tile n: O / den -> 16-bit -> global memory
            gsub += it.nsub;
            const int gl = gsub - 1;
            {
                int f = 0;
                if (!mbar_wait_abortable(&c->den_full, n & 1, s_abort)) f = kStatusP2Den;
                else if (!mbar_wait_abortable(c->pv_done + (gl & 1), (gl >> 1) & 1, s_abort)) f = kStatusP2PvDone;
                if (f) fail = f;
                if (group_failed()) break;
            }
            tc_fence_after();
            const float inv_den = 1.f / c->den[r];
            const int row = it.m0 + r;
            T* orow = reinterpret_cast<T*>(a.out) + static_cast<long long>(it.b) * a.o_sb +
                      static_cast<long long>(it.h) * a.o_sh + static_cast<long long>(row) * a.o_ss;
            // The whole row is converted into registers first (256 16-bit values = 128 registers) so that the
            // TMEM columns are released after eight loads; the global stores follow.
            uint32_t packed[D / 2];
#pragma unroll
            for (int q4 = 0; q4 < D / 32; ++q4) {
                uint32_t o[32];
                tmem_ld32(lane_base + kColO + q4 * 32, o);
                tmem_wait_ld();
#pragma unroll
                for (int i = 0; i < 16; ++i)
                    packed[q4 * 16 + i] = Num<T>::pack(__uint_as_float(o[2 * i]) * inv_den, __uint_as_float(o[2 * i + 1]) * inv_den);
            }
            // the output (and the row sums) of this tile have been read: its successor may overwrite them
            tc_fence_before();
            __syncwarp();
            if (lane == 0) {
                remote_arrive_relaxed(map_to_cta(&c->o_free, 0));
                mbar_arrive(&c->den_free);
            }
            if (row < a.S) {
#pragma unroll
                for (int ch = 0; ch < D / 8; ++ch)
                    *reinterpret_cast<uint4*>(orow + ch * 8) =
                        make_uint4(packed[ch * 4 + 0], packed[ch * 4 + 1], packed[ch * 4 + 2], packed[ch * 4 + 3]);
            }
            cur = nxt;
        }
        if (fail) give_up(fail);
    }
    else {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 128;");
        if (warp == 8) {
            // ============================================ K/V producer
            if (elect_one()) {
                int s = 0;            // ring stage of the next tile
                uint32_t epar = 1;    // parity to wait for on the stage's empty barrier (passes at once on the first turn)
                const int r0 = static_cast<int>(rank);
                const uint32_t full0 = map_to_cta(c->kv_full, 0);
                // next tile of the consumption order, this CTA's half of it
                auto next_stage = [&]() -> uint8_t* {
                    if (!mbar_wait_abortable(c->kv_empty + s, epar, s_abort)) { fail = kStatusP2KvEmpty; return nullptr; }
                    remote_expect_tx(full0 + 8 * s, kPrStageBytes);
                    ++kv_issued;
                    return smem_kv + s * kPrStageBytes;
                };
                auto emit_k = [&](int j, const P2Item& it) {  // 32 of the 64 keys, all columns
                    uint8_t* dst = next_stage();
                    if (dst == nullptr) return;
#pragma unroll
                    for (int bx = 0; bx < NB; ++bx)
                        tma_load_4d_pair(dst + bx * kPrKBoxBytes, &tm_k, full0 + 8 * s, bx * 64, j * kSub + r0 * (kSub / 2),
                                         it.kh, it.b);
                    if (++s == kPrRing) { s = 0; epar ^= 1; }
                };
                auto emit_v = [&](int j, const P2Item& it) {  // all 64 keys, half of the columns
                    uint8_t* dst = next_stage();
                    if (dst == nullptr) return;
#pragma unroll
                    for (int bx = 0; bx < NB / 2; ++bx)
                        tma_load_4d_pair(dst + bx * kPrVBoxBytes, &tm_v, full0 + 8 * s, r0 * (D / 2) + bx * 64, j * kSub, it.kh,
                                         it.b);
                    if (++s == kPrRing) { s = 0; epar ^= 1; }
                };
                // (see attn_fwd_persist.cuh: the first K copy waits for the row-prepare this grid may depend on)
                grid_dep_wait();
                int n = 0;
                for (; !fail; ++n) {
                    const int idx = pr_take_item(c, n, fail);
                    if (idx < 0) break;
                    const P2Item it = pr_decode(idx, rank, a);
                    emit_k(0, it);
                    for (int jj = 0; jj < it.nsub && !fail; ++jj) {
                        if (jj + 1 < it.nsub) emit_k(jj + 1, it);
                        if (!fail) emit_v(jj, it);
                    }
                }
                if (fail) give_up(fail);
                if (!leader) drain_mma(n, kv_issued, fail != 0);
                remote_store(map_to_cta(c->issued + rank, 0), kv_issued);
            }
        } else if (warp == 9 && leader) {
            // ============================================ MMA issuer of the pair
            if (elect_one()) {
                const uint32_t kv_addr = smem_u32(smem_kv);
                const uint64_t k_desc = umma_desc_sw128(0, 16, 1024);              // K-major operand (K)
                const uint64_t v_desc = umma_desc_sw128(0, kPrVBoxBytes, 1024);    // MN-major operand (V), 8 KB between column boxes
                const uint32_t k_hi = static_cast<uint32_t>(k_desc >> 32), v_hi = static_cast<uint32_t>(v_desc >> 32);
                const uint32_t k_lo = static_cast<uint32_t>(k_desc) | ((kv_addr & 0x3FFFFu) >> 4);
                const uint32_t v_lo = static_cast<uint32_t>(v_desc) | ((kv_addr & 0x3FFFFu) >> 4);
                auto issue_qk = [&](int stage, int buf) {
                    const uint32_t ka = k_lo + stage * (kPrStageBytes >> 4);
                    const uint32_t d = tmem_base + buf * kSub;
#pragma unroll
                    for (int ks = 0; ks < D / 16; ++ks)
                        umma_ts_pair_lohi(d, tmem_base + kColQ + ks * 8, ka + (ks / 4) * (kPrKBoxBytes >> 4) + (ks % 4) * 2, k_hi,
                                          kIdescQK, ks > 0 ? 1u : 0u);
                };
                auto issue_pv = [&](int stage, int buf, uint32_t accumulate) {
                    const uint32_t va = v_lo + stage * (kPrStageBytes >> 4);
                    const uint32_t d = tmem_base + kColO;
                    const uint32_t pa = tmem_base + buf * kSub;
                    umma_ts_pair_lohi(d, pa, va, v_hi, kIdescPV, accumulate);
#pragma unroll
                    for (int ks = 1; ks < kSub / 16; ++ks) umma_ts_pair_lohi(d, pa + ks * 8, va + ks * 128, v_hi, kIdescPV, 1u);
                };
                int st = 0;
                uint32_t par = 0;
                uint32_t nq = 0, np = 0;
                // scores of sub-block j of the running tile; the tile's last one also reports "every Q K^T done"
                auto take_k = [&](bool last) {
                    if (!mbar_wait_abortable(c->kv_full + st, par, s_abort)) { fail = kStatusP2KvFull; return; }
                    tc_fence_after();
                    issue_qk(st, nq & 1);
                    umma_commit_pair(c->s_full + (nq & 1));
                    ++nq;
                    umma_commit_pair(c->kv_empty + st);
                    if (last) umma_commit_pair(&c->qk_done);
                    if (++st == kPrRing) { st = 0; par ^= 1; }
                };
                int n = 0;
                for (; !fail; ++n) {
                    const int idx = pr_take_item(c, n, fail);
                    if (idx < 0) break;
                    const P2Item it = pr_decode(idx, rank, a);
                    if (!mbar_wait_abortable(&c->q_ready, n & 1, s_abort)) { fail = kStatusP2QReady; break; }
                    take_k(it.nsub == 1);
                    for (int jj = 0; jj < it.nsub && !fail; ++jj) {
                        if (jj + 1 < it.nsub) {
                            take_k(jj + 2 == it.nsub);
                            if (fail) break;
                        }
                        // ---- O += P V of sub-block jj
                        if (!mbar_wait_abortable(c->kv_full + st, par, s_abort)) { fail = kStatusP2KvFull; break; }
                        // the first P V of a tile overwrites the previous tile's output: the epilogue must have read it
                        if (jj == 0 && n > 0 && !mbar_wait_abortable(&c->o_free, (n - 1) & 1, s_abort)) { fail = kStatusP2OFree; break; }
                        if (!mbar_wait_abortable(c->p_ready + (np & 1), (np >> 1) & 1, s_abort)) { fail = kStatusP2PReady; break; }
                        tc_fence_after();
                        issue_pv(st, np & 1, jj > 0 ? 1u : 0u);
                        umma_commit_pair(c->pv_done + (np & 1));
                        ++np;
                        umma_commit_pair(c->kv_empty + st);
                        if (++st == kPrRing) { st = 0; par ^= 1; }
                    }
                }
                if (fail) give_up(fail);
                if (nq > 0) {  // (else nothing was issued; CTA 1's wait then runs out)
                    umma_commit_pair(&c->mma_done);
                    drain_mma(n, static_cast<int>(nq + np), fail != 0);
                }
            }
        } else if (warp == 10) {
            // ============================================ scheduler (CTA 0) and raw-Q producer
            if (elect_one()) {
                for (int n = 0; !fail; ++n) {
                    if (leader) {
                        // the first item needs no counter; later ones are claimed when the running one is about to
                        // finish (its softmax group says so), so that no pair sits on work it cannot start yet
                        if (n > 0 && !mbar_wait_abortable(&c->near_end, (n - 1) & 1, s_abort)) { fail = kStatusP2Item; break; }
                        const int pairs = static_cast<int>(gridDim.x / 2);
                        const int nxt = n == 0 ? static_cast<int>(blockIdx.x / 2) : pairs + static_cast<int>(atomicAdd(a.sched, 1u));
                        const int idx = nxt < n_items ? nxt : -1;
                        const int rs = n & (kPrItemRing - 1);
                        *reinterpret_cast<volatile int*>(c->item + rs) = idx;
                        mbar_arrive(c->item_full + rs);
                        remote_store(map_to_cta(c->item + rs, 1), idx);
                        remote_arrive(map_to_cta(c->item_full + rs, 1));
                    }
                    const int idx = pr_take_item(c, n, fail);
                    if (idx < 0) break;
                    const P2Item it = pr_decode(idx, rank, a);
                    // the Q buffer is free once the previous tile's prepared Q has been copied into TMEM
                    if (n > 0 && !mbar_wait_abortable(&c->q_free, (n - 1) & 1, s_abort)) { fail = kStatusP2QFree; break; }
                    mbar_expect_tx(&c->q_full, kP2QBytes);
#pragma unroll
                    for (int bx = 0; bx < NB; ++bx) tma_load_4d(smem_q + bx * kBoxBytes, &tm_q, &c->q_full, bx * 64, it.m0, it.h, it.b);
                    q_issued = n + 1;
                }
                if (fail) give_up(fail);
            }
        }
    }

    // ---- common exit
    __syncwarp();
    tc_fence_before();
    cluster_sync();  // every role of both CTAs has ended (and a failure of either shows in both)
    if (!dead && *s_abort != 0) {
        // Leave no copy in flight.  Both CTAs' K/V copies complete on CTA 0's barriers: arrivals that a CTA did not make
        // are made up for, so that every phase ends with the copies that were issued.
        if (leader && warp == 8 && elect_one()) {
            volatile int* issued = c->issued;
            const int lo = min(issued[0], issued[1]), hi = max(issued[0], issued[1]);
            for (int i = lo; i < hi; ++i) mbar_arrive(c->kv_full + i % kPrRing);
            for (int i = 0; i < kPrRing; ++i)
                if (hi > i) mbar_wait(c->kv_full + i, ((hi - 1 - i) / kPrRing) & 1);
        }
        if (warp == 10 && elect_one() && q_issued > 0) mbar_wait(&c->q_full, (q_issued - 1) & 1);
    }
    __syncthreads();
    cluster_sync();  // no copy, MMA, commit or remote arrival of the pair is under way any more
    if (warp == 0) tmem_dealloc_pair(tmem_base, kTmemCols);
    // The last CTA to leave resets the work counter for the next launch that uses it.
    if (tid == 0) {
        __threadfence();
        const unsigned int left = atomicAdd(a.sched + 1, 1u);
        if (left == gridDim.x - 1) {
            a.sched[0] = 0;
            a.sched[1] = 0;
            __threadfence();
        }
    }
    cluster_sync();
}

}  // namespace kf
