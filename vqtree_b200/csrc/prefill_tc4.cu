// Fused VQ-attention prefill on the sm_100a tensor cores, one softmax thread per query row, in two forms (KEYS):
//   128   one CTA per SM, steps of 128 keys, three softmax warpgroups;
//   64    two CTAs per SM, steps of 64 keys, two softmax warpgroups each: short tiles on grids that fill the chip (see
//         launch_keys for where the line lies).
//
// One CTA owns one 128-row query tile of one (batch, query head) and walks its work items (far
// codebook tiles, boundary block, interior blocks, causal diagonal - see TcWork) with ONE online
// softmax (this replaces the reference's two kernels and their log-sum-exp merge,
// ops/triton_fused_vq_attn.py:202-250).  An item of 128 keys is one step, or two of 64.  Tensor memory (all 512
// columns, or 256 per CTA): the S/P buffers, one per warpgroup, KEYS columns each, and the O accumulator.  Roles:
//   softmax     warpgroup g = warp / 4 owns score buffer g and takes the steps j = g, g + 3, ... (g, g + 2, ...: half g of
//               every item); inside it one thread per query row reads the row's scores 64 at a time, so the row maximum
//               and the row sum need no exchange.  All rows of the tile share one reference maximum
//               per row, kept in shared memory and handed from step j to step j+1 through a
//               barrier chain: the thread of step j picks up the reference left by step j-1, raises
//               it only when its item's maximum is more than 2^8 above it (then it rescales O once the
//               product of step j-1 has finished), publishes it, and only then exponentiates - so
//               the warpgroups exponentiate their steps at the same time.
//               Each thread keeps the partial denominator of its own steps, scaled to the reference
//               it used last; the partial sums are merged at the end.
//   next warp   one thread issues every tcgen05.mma: S(j) = Q K(j)^T three (two) steps ahead (operands in
//               shared memory), O += P(j) V(j) (P from tensor memory, V MN-major in shared memory);
//   last warp   one thread issues the TMA tile loads into a ring of KEYS-row slots in the order the
//               tensor pipe consumes them (K0 K1 K2 V0 K3 V1 ...).  ReRoPE: both kinds of queries are resident (128), or
//               the query tile holds the constant-position queries first (far tiles, boundary block) and is reloaded with
//               the rotated ones once the last score product that reads it has finished (64: shared memory for one).
// What bounds it: no single unit, but the hand-offs of a step and, on short tiles, start and end of a CTA.  The 128-key form
// reads a row's scores as two batches of 64 (one wait for each; four batches of 32: 1.24 -> 1.30 ms, B1 H32 L32768 W1024 MK1024, plain
// RoPE, in turn on one card) in 128 registers without spills; the 64-key form is held to 96 registers by its two CTAs and spills
// 64 - 76 bytes a thread.  128 / 64 keys in turn on one card: that shape 1.17 / 1.24 ms; ReRoPE, B2 L16384 W512 MK2048 1.68 /
// 1.78 ms; half, ReRoPE, L5001, MK1024 206 / 209 us.
// Hand-offs are mbarriers (tcgen05.commit arrives for the MMA side); every wait is bounded and a
// failed wait raises the status word; all roles meet at one final barrier and TMEM is freed.
#include "prefill_tc_common.cuh"

namespace vq {

using namespace ptx;

constexpr float kT4Lazy = 8.f;    // log2 units: P stays below 2^8

// KEYS: keys per step, 64 (two CTAs per SM) or 128 (one)
template <int D, int KEYS>
struct T4Cfg {
    static constexpr int kCtas = KEYS == 64 ? 2 : 1;          // per SM
    static constexpr int kBufs = KEYS == 64 ? 2 : 3;          // S/P buffers = softmax warpgroups
    static constexpr int kSteps = kBlock / KEYS;              // steps per item
    static constexpr int kWarps = 4 * kBufs;                  // softmax warps
    static constexpr int kWarpMma = kWarps, kWarpTma = kWarps + 1;
    static constexpr int kThreads = (kWarps + 2) * 32;
    static constexpr int NH = D / 64;
    static constexpr int kHalf = KEYS * 128;                  // one TMA box of K / V: KEYS rows x 64 columns
    static constexpr int kQTile = NH * kHalfBytes;            // 128 x D
    static constexpr int kQTiles = KEYS == 64 ? 1 : 2;        // 2: both kinds of queries resident, 1: reloaded
    static constexpr int kTile = NH * kHalf;                  // KEYS x D
    static constexpr int kSlots = KEYS == 64 ? 4 : 3;         // ring of K / V tiles: with the query tiles what fits into the CTA's share
    static constexpr int kQ = 0, kRing = kQTiles * kQTile;
    static constexpr int kTotal = kRing + kSlots * kTile + 1024;  // + slack for 1024-byte alignment
    static constexpr uint32_t kColS = 0, kColO = KEYS * kBufs, kCols = KEYS == 64 ? 256 : 512;
    static constexpr int kOq = D / 2;                          // O columns written by one thread at the end
};

// scores of 64 columns outside [lo, hi) of the step: excluded
__device__ __forceinline__ void t4_mask_range(uint32_t (&r)[64], int lo, int hi)
{
#pragma unroll
    for (int c = 0; c < 64; ++c)
        if (c < lo || c >= hi) r[c] = 0xff800000u;
}

// Far tile with empty codes: a code with cnt == 0 is excluded from the maximum and from P, as the reference does before its
// maximum (ops/triton_fused_vq_attn.py:44-46) - otherwise an unused codeword with a dominating score could push every real
// weight below the exponent range.  cw: the counts of the step's 64 columns.
__device__ __forceinline__ void t4_mask_empty(uint32_t (&r)[64], const float *cw)
{
#pragma unroll
    for (int c = 0; c < 64; c += 4) {
        const float4 w = *reinterpret_cast<const float4 *>(cw + c);
        if (!(w.x > 0.f)) r[c] = 0xff800000u;
        if (!(w.y > 0.f)) r[c + 1] = 0xff800000u;
        if (!(w.z > 0.f)) r[c + 2] = 0xff800000u;
        if (!(w.w > 0.f)) r[c + 3] = 0xff800000u;
    }
}

__device__ __forceinline__ float t4_max(const uint32_t (&r)[64])
{
    float mx[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
    for (int j = 0; j < 32; ++j) mx[j & 3] = fmax3(mx[j & 3], __uint_as_float(r[2 * j]), __uint_as_float(r[2 * j + 1]));
    return fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3]));
}

// P = exp2(S * scale - m) of the 64 scores, packed 16-bit floats written to the 32 columns at p_addr; returns
// sum plus the (FAR: count-weighted) sums of the two halves, one after the other.
template <bool FAR, bool F16>
__device__ __forceinline__ float t4_exp(const uint32_t (&r)[64], uint32_t p_addr, const float *cw, float scale_log2, float neg_m, float sum)
{
#pragma unroll
    for (int half = 0; half < 2; ++half) {
        float ls[4] = {0.f, 0.f, 0.f, 0.f};
        uint32_t pk[16];
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const int c = 32 * half + 4 * j;
            float w[4] = {1.f, 1.f, 1.f, 1.f};
            if (FAR) {
                const float4 w4 = *reinterpret_cast<const float4 *>(cw + c);
                w[0] = w4.x; w[1] = w4.y; w[2] = w4.z; w[3] = w4.w;
            }
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                float t0, t1;
                ffma2(t0, t1, __uint_as_float(r[c + 2 * i]), __uint_as_float(r[c + 2 * i + 1]), scale_log2, scale_log2, neg_m, neg_m);
                const float p0 = ex2(t0), p1 = ex2(t1);
                if (FAR) ffma2(ls[2 * i], ls[2 * i + 1], p0, p1, w[2 * i], w[2 * i + 1], ls[2 * i], ls[2 * i + 1]);
                else fadd2(ls[2 * i], ls[2 * i + 1], ls[2 * i], ls[2 * i + 1], p0, p1);
                pk[2 * j + i] = pack16<F16>(p0, p1);
            }
        }
        tmem_st16(p_addr + 16 * half, pk);
        sum += (ls[0] + ls[1]) + (ls[2] + ls[3]);
    }
    return sum;
}

// One row's scores of 64 columns, those of excluded keys set to -inf.  lo, hi: valid columns of the 64 (kDiag, kBdA, kBdB).
__device__ __forceinline__ void t4_scores(uint32_t s_addr, int kind, bool has_empty, int lo, int hi, const float *cw, uint32_t (&r)[64])
{
    tmem_ld32(s_addr, *reinterpret_cast<uint32_t(*)[32]>(&r[0]));
    tmem_ld32(s_addr + 32, *reinterpret_cast<uint32_t(*)[32]>(&r[32]));
    tc_wait_ld();
    if (kind == kFar) {
        if (has_empty) t4_mask_empty(r, cw);
    } else if (kind != kFull) {
        t4_mask_range(r, lo, hi);
    }
}

template <int D, bool F16, int KEYS>
__global__ void __launch_bounds__(T4Cfg<D, KEYS>::kThreads, T4Cfg<D, KEYS>::kCtas)
prefill_tc4_kernel(const __grid_constant__ CUtensorMap tm_q1, const __grid_constant__ CUtensorMap tm_q2,
                   const __grid_constant__ CUtensorMap tm_k1, const __grid_constant__ CUtensorMap tm_k3,
                   const __grid_constant__ CUtensorMap tm_v, const __grid_constant__ CUtensorMap tm_cb,
                   const __grid_constant__ CUtensorMap tm_vs, TcParams p)
{
    using C = T4Cfg<D, KEYS>;
    constexpr int NH = C::NH, NS = C::kSlots, NB3 = C::kBufs, SPI = C::kSteps;
    extern __shared__ uint8_t smem_raw[];
    uint8_t *smem = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    __shared__ __align__(8) uint64_t bar_q, q_free, kv_full[NS], kv_empty[NS], s_full[NB3], p_full[NB3], pv_done[NB3], refbar[NB3][4], halfbar[4], endbar;
    __shared__ uint32_t s_tmem;
    __shared__ int s_err;
    __shared__ __align__(16) float s_cw[C::kWarps][KEYS];  // [softmax warp][column]: counts of the far step it works on
    __shared__ float s_ref[kBlock];                          // reference maximum of every query row (log2 units)
    __shared__ float s_half[SPI == 2 ? kBlock : 1];          // maximum of every row over the second half of an item
    __shared__ float s_lend[NB3][kBlock], s_mend[NB3][kBlock];  // partial denominators and the references they are scaled to

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    // grid.x = (query tile, query head inside its kv-head group), grid.y = (batch, kv head): the query heads
    // that share a kv head run next to each other, so their K / V / value-sum tiles meet in L2
    const int G = p.Hq / p.Hkv;
    const int m = p.ntiles - 1 - static_cast<int>(blockIdx.x) / G;  // heavy tiles first
    const int u = blockIdx.y;
    const int b = u / p.Hkv, hk = u % p.Hkv;
    const int hq = hk * G + static_cast<int>(blockIdx.x) % G;
    const int bh = b * p.Hq + hq;
    const TcWork work(p, m);
    const int n = SPI * work.n_items;                        // steps: part s % SPI of item s / SPI
    const int n_q2 = p.rerope ? SPI * (work.n_far + (work.n_bd == 2 ? 1 : 0)) : 0;   // steps scored with q2 come first

    if (tid == 0) {
        mbar_init(&bar_q, 1);
        mbar_init(&q_free, 1);
        for (int i = 0; i < NS; ++i) {
            mbar_init(&kv_full[i], 1);
            mbar_init(&kv_empty[i], 1);
        }
        for (int i = 0; i < NB3; ++i) {
            mbar_init(&s_full[i], 1);
            mbar_init(&p_full[i], 4);  // one arrival per warp of the warpgroup
            mbar_init(&pv_done[i], 1);
            for (int g = 0; g < 4; ++g) mbar_init(&refbar[i][g], 1);
        }
        for (int g = 0; g < 4; ++g) mbar_init(&halfbar[g], 1);
        mbar_init(&endbar, C::kWarps);
        fence_mbar_init();
        s_err = 0;
    }
    if (tid < kBlock) s_ref[tid] = -INFINITY;
    if (warp == C::kWarpTma) {
        __syncwarp();
        tmem_alloc(&s_tmem, C::kCols);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = s_tmem;

    if (warp == C::kWarpTma) {
        // ================================================================== TMA producer
        if (elect_one()) {
            prefetch_tmap(&tm_q1); prefetch_tmap(&tm_k1); prefetch_tmap(&tm_v);
            auto load_q = [&](const CUtensorMap *tm, int tile) {
#pragma unroll
                for (int h = 0; h < NH; ++h) tma_load_4d(smem + C::kQ + tile * C::kQTile + h * kHalfBytes, tm, &bar_q, 64 * h, m * kBlock, hq, b);
            };
            if constexpr (C::kQTiles == 2) {
                mbar_expect_tx(&bar_q, (n_q2 > 0 ? 2 : 1) * C::kQTile);
                load_q(&tm_q1, 0);
                if (n_q2 > 0) load_q(&tm_q2, 1);
            } else {
                mbar_expect_tx(&bar_q, C::kQTile);
                load_q(n_q2 > 0 ? &tm_q2 : &tm_q1, 0);
            }
            bool ok = true;
            int slot = 0;               // ring slot of the next load (consumption sequence K0 K1 V0 K2 V1 ...)
            uint32_t free_par = 1u;     // phase of kv_empty[slot] that frees it; the first round needs no wait
            bool first_round = true;
            auto load = [&](int step, bool is_v) {
                if (!ok) return;
                if (C::kQTiles == 1 && !is_v && step == n_q2 && n_q2 > 0) {   // the query tile changes once its last score product has finished
                    if (!mbar_wait(&q_free, 0, p.wait_limit)) {
                        ok = false;
                        return;
                    }
                    mbar_expect_tx(&bar_q, C::kQTile);
                    load_q(&tm_q1, 0);
                }
                if (!first_round && !mbar_wait(&kv_empty[slot], free_par, p.wait_limit)) {
                    ok = false;
                    return;
                }
                const int it = step / SPI, kind = work.kind(it), row0 = work.block(it) * kBlock + (step % SPI) * KEYS;
                uint8_t *dst = smem + C::kRing + slot * C::kTile;
                mbar_expect_tx(&kv_full[slot], C::kTile);
#pragma unroll
                for (int h = 0; h < NH; ++h) {
                    if (kind == kFar) {
                        if (is_v) tma_load_3d(dst + h * C::kHalf, &tm_vs, &kv_full[slot], 64 * h, row0, u * p.NB + work.far_blk);
                        else tma_load_3d(dst + h * C::kHalf, &tm_cb, &kv_full[slot], 64 * h, row0, hk);
                    } else {
                        const CUtensorMap *tm = is_v ? &tm_v : (kind == kBdA ? &tm_k3 : &tm_k1);
                        tma_load_4d(dst + h * C::kHalf, tm, &kv_full[slot], 64 * h, row0, hk, b);
                    }
                }
                if (++slot == NS) {
                    slot = 0;
                    free_par ^= 1u;
                    first_round = false;
                }
            };
            for (int j = 0; j < NB3 && j < n; ++j) load(j, false);
            for (int j = 0; j < n; ++j) {
                load(j, true);
                if (j + NB3 < n) load(j + NB3, false);
            }
            if (!ok) s_err = 1;
        }
    } else if (warp == C::kWarpMma) {
        // ================================================================== MMA issuer
        // The tensor pipe's queue is shallow: whatever this thread does between two groups of MMAs is time the
        // pipe idles.  So the loop carries no divisions and no per-item classification: ring slot, score buffer and
        // their barrier phases are running counters, an operand's descriptor is a base built once plus the slot's
        // offset, and a step needs the constant-position query exactly when it comes before `n_q2`.
        if (elect_one()) {
            constexpr uint32_t idesc_qk = idesc_f16kind(128, KEYS, 0, 0, F16 ? 0u : 1u);
            constexpr uint32_t idesc_pv = idesc_f16kind(128, D, 0, 1, F16 ? 0u : 1u);
            const uint64_t d_q = smem_desc_sw128(smem_u32(smem + C::kQ), 16, 1024);
            const uint64_t d_k0 = smem_desc_sw128(smem_u32(smem + C::kRing), 16, 1024);          // K tiles: K-major
            const uint64_t d_v0 = smem_desc_sw128(smem_u32(smem + C::kRing), C::kHalf, 1024);    // V tiles: MN-major
            bool ok = mbar_wait(&bar_q, 0, p.wait_limit);
            int slot = 0;
            uint32_t slot_par = 0;                 // phase of the ring slot about to be consumed
            int sbuf = 0, pbuf = 0;                // score buffer of the next S product / of the next P V product
            uint32_t p_par = 0;                    // phase of p_full[pbuf]
            auto next_slot = [&]() {
                if (++slot == NS) {
                    slot = 0;
                    slot_par ^= 1u;
                }
            };
            auto qk = [&](int it) {  // S(it) = Q K(it)^T into the next score buffer (free: its previous product was issued before)
                if (!ok) return;
                if ((C::kQTiles == 1 && it == n_q2 && it > 0 && !mbar_wait(&bar_q, 1, p.wait_limit)) || !mbar_wait(&kv_full[slot], slot_par, p.wait_limit)) {
                    ok = false;
                    return;
                }
                tc_fence_after();
                const uint64_t db = d_k0 + static_cast<uint64_t>((slot * C::kTile) >> 4);
                const uint64_t da = d_q + static_cast<uint64_t>(((C::kQTiles == 2 && it < n_q2 ? C::kQTile : 0)) >> 4);
                const uint32_t sdst = tmem + C::kColS + KEYS * sbuf;
#pragma unroll
                for (int h = 0; h < NH; ++h)
#pragma unroll
                    for (int k4 = 0; k4 < 4; ++k4) {
                        constexpr int kStep = 32 >> 4;
                        const uint64_t qa = da + static_cast<uint64_t>(((h * kHalfBytes) >> 4) + k4 * kStep);
                        const uint64_t kb = db + static_cast<uint64_t>(((h * C::kHalf) >> 4) + k4 * kStep);
                        if (h == 0 && k4 == 0) mma_ss_first(sdst, qa, kb, idesc_qk);
                        else mma_ss_acc(sdst, qa, kb, idesc_qk);
                    }
                tc_commit(&kv_empty[slot]);
                tc_commit(&s_full[sbuf]);
                if (C::kQTiles == 1 && it + 1 == n_q2) tc_commit(&q_free);
                next_slot();
                if (++sbuf == NB3) sbuf = 0;
            };
            auto pv = [&](int it) {  // O += P(it) V(it)
                if (!ok) return;
                if (!mbar_wait(&p_full[pbuf], p_par, p.wait_limit) || !mbar_wait(&kv_full[slot], slot_par, p.wait_limit)) {
                    ok = false;
                    return;
                }
                tc_fence_after();
                const uint64_t dv = d_v0 + static_cast<uint64_t>((slot * C::kTile) >> 4);
                const uint32_t odst = tmem + C::kColO, psrc = tmem + C::kColS + KEYS * pbuf;
                if (it == 0) mma_ts_first(odst, psrc, dv, idesc_pv);
                else mma_ts_acc(odst, psrc, dv, idesc_pv);
#pragma unroll
                for (int kk = 1; kk < KEYS / 16; ++kk)  // keys 16 kk ..: packed 16-bit P over the first half of the score buffer
                    mma_ts_acc(odst, psrc + 8 * kk, dv + static_cast<uint64_t>((kk * 2048) >> 4), idesc_pv);
                tc_commit(&kv_empty[slot]);
                tc_commit(&pv_done[pbuf]);
                next_slot();
                if (++pbuf == NB3) {
                    pbuf = 0;
                    p_par ^= 1u;
                }
            };
            for (int j = 0; j < NB3 && j < n; ++j) qk(j);
            for (int j = 0; j < n; ++j) {
                pv(j);
                if (j + NB3 < n) qk(j + NB3);
            }
            if (!ok) s_err = 1;
        }
    } else {
        // ================================================================== softmax
        constexpr unsigned kAll = 0xffffffffu;
        const int g = warp >> 2, lq = warp & 3;           // warpgroup (= score buffer) and lane quarter (32 query rows)
        const int row = lq * 32 + lane;                   // query row inside the tile (= TMEM lane)
        const uint32_t lane_off = static_cast<uint32_t>(lq * 32) << 16;
        const uint32_t sa = tmem + lane_off + C::kColS + KEYS * g;
        const uint32_t o_addr = tmem + lane_off + C::kColO;
        float my_ref = -INFINITY, l_part = 0.f;           // l_part: sum over this thread's steps, scaled to my_ref
        bool ok = true;
        // Counts of a far step (its columns begin at KEYS * step): lane l fetches those of columns l, 32 + l, ... one of
        // the warp's steps ahead; the warp keeps them in its own shared-memory row.
        constexpr int NCW = KEYS / 32;
        const int far_steps = SPI * work.n_far;
        const float *cnt_base = p.cnt + (static_cast<int64_t>(u) * p.NB + work.far_blk) * p.MK + lane;
        float *cw = &s_cw[warp][0];
        float cnt_reg[NCW];
#pragma unroll
        for (int i = 0; i < NCW; ++i) cnt_reg[i] = g < far_steps ? __ldg(cnt_base + g * KEYS + 32 * i) : 0.f;
#pragma unroll 1
        for (int it = g; it < n; it += NB3) {                 // `it` counts steps
            const int par = (it / NB3) & 1;
            const int kind = work.kind(it / SPI);
            const int c0 = KEYS * (it % SPI);             // first of the item's columns
            bool has_empty = false;                       // warp-uniform: some code of this far step has no member
            if (kind == kFar) {
                __syncwarp();
                bool full = true;
#pragma unroll
                for (int i = 0; i < NCW; ++i) {
                    cw[32 * i + lane] = cnt_reg[i];
                    full = full && cnt_reg[i] > 0.f;
                }
                has_empty = __any_sync(kAll, !full);
                __syncwarp();
                if (it + NB3 < far_steps) {
#pragma unroll
                    for (int i = 0; i < NCW; ++i) cnt_reg[i] = __ldg(cnt_base + (it + NB3) * KEYS + 32 * i);
                }
            }
            // valid key columns of this row
            const int lo = kind == kBdB ? row - c0 : 0, hi = kind == kDiag ? row + 1 - c0 : kind == kBdA ? row - c0 : KEYS;
            if (!__all_sync(kAll, mbar_wait(&s_full[g], par, p.wait_limit))) {
                ok = false;
                break;
            }
            tc_fence_after();
            // ---- the row's scores and their maximum (64 stay in registers, of 128 the second pass reads them again)
            uint32_t r[64];
            float mx = -INFINITY;
#pragma unroll
            for (int c = 0; c < KEYS; c += 64) {
                t4_scores(sa + c, kind, has_empty, lo - c, hi - c, cw + c, r);
                mx = fmaxf(mx, t4_max(r));
            }
            float m_tile = mx * p.scale_log2;
            if (SPI == 2 && g == 1) {                     // the other half's thread of this row may want it
                s_half[row] = m_tile;
                __syncwarp();
                if (lane == 0) mbar_arrive(&halfbar[lq]);
            }
            // ---- the reference left by the previous step; raise it only when this item is far above it
            if (it > 0 && !__all_sync(kAll, mbar_wait(&refbar[(g + NB3 - 1) % NB3][lq], ((it - 1) / NB3) & 1, p.wait_limit))) {
                ok = false;
                break;
            }
            const float ref = s_ref[row];
            if (SPI == 2 && g == 0 && __any_sync(kAll, m_tile > ref + kT4Lazy || ref == -INFINITY)) {
                // A raised reference is the maximum over the whole item: the weight of the largest score is then exactly
                // one and not rounded (left at the maximum of half an item, the output was 0.5 - 0.9 % further from the
                // 64-bit result).  The second half's scores do not depend on anything this thread has yet to do, and its
                // maximum is not overwritten before the arrival at refbar below.
                if (!__all_sync(kAll, mbar_wait(&halfbar[lq], par, p.wait_limit))) {
                    ok = false;
                    break;
                }
                m_tile = fmaxf(m_tile, s_half[row]);
            }
            float m_use = ref;
            if (m_tile > ref + kT4Lazy || ref == -INFINITY) m_use = fmaxf(ref, m_tile);
            if (m_use != ref) s_ref[row] = m_use;
            __syncwarp();
            if (lane == 0) mbar_arrive(&refbar[g][lq]);   // the warp's 32 stores are ordered before it
            const float m_safe = (m_use == -INFINITY) ? 0.f : m_use;
            // a row without any valid key so far has an all-zero O row: nothing to rescale
            const bool rescale = (m_use != ref) && (ref != -INFINITY);
            if (__any_sync(kAll, rescale)) {
                // O may be touched once the product of the previous item has finished (it >= 1 here)
                if (!__all_sync(kAll, mbar_wait(&pv_done[(it - 1) % NB3], ((it - 1) / NB3) & 1, p.wait_limit))) {
                    ok = false;
                    break;
                }
                tc_fence_after();
                const float alpha = rescale ? ex2(ref - m_safe) : 1.f;
#pragma unroll
                for (int c = 0; c < D / 16; ++c) {
                    uint32_t o[16];
                    tmem_ld16(o_addr + 16 * c, o);
                    tc_wait_ld();
#pragma unroll
                    for (int j = 0; j < 16; ++j) o[j] = __float_as_uint(__uint_as_float(o[j]) * alpha);
                    tmem_st16(o_addr + 16 * c, o);
                }
            }
            if (my_ref != m_use) {
                l_part *= ex2(my_ref - m_safe);           // my_ref = -inf: l_part is 0 and stays 0
                my_ref = m_use;
            }
            // ---- exponentials; P goes over the first half of the score columns, never ahead of a read
            float ls = 0.f;
#pragma unroll
            for (int c = 0; c < KEYS; c += 64) {
                if (KEYS > 64) t4_scores(sa + c, kind, has_empty, lo - c, hi - c, cw + c, r);
                ls = kind == kFar ? t4_exp<true, F16>(r, sa + c / 2, cw + c, p.scale_log2, -m_safe, ls)
                                  : t4_exp<false, F16>(r, sa + c / 2, cw + c, p.scale_log2, -m_safe, ls);
            }
            l_part += ls;
            tc_wait_st();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&p_full[g]);
        }
        // ---- epilogue: merge the partial denominators, O / l once the last product has finished
        s_lend[g][row] = l_part;
        s_mend[g][row] = my_ref;
        __syncwarp();
        if (lane == 0) mbar_arrive(&endbar);
        if (ok && !__all_sync(kAll, mbar_wait(&endbar, 0, p.wait_limit))) ok = false;
        if (ok && !__all_sync(kAll, mbar_wait(&pv_done[(n - 1) % NB3], ((n - 1) / NB3) & 1, p.wait_limit))) ok = false;
        tc_fence_after();
        if (!ok) s_err = 1;
        if (ok && g < 2) {
            const float ref = s_ref[row];
            float den = 0.f;
#pragma unroll
            for (int i = 0; i < NB3; ++i) {
                const float li = s_lend[i][row];
                if (li > 0.f) den += li * ex2(s_mend[i][row] - ref);
            }
            const float inv = den > 0.f ? 1.f / den : 0.f;
            const int64_t grow = static_cast<int64_t>(m) * kBlock + row;
            uint32_t r[C::kOq];
#pragma unroll
            for (int c = 0; c < C::kOq / 32; ++c) tmem_ld32(o_addr + g * C::kOq + 32 * c, *reinterpret_cast<uint32_t(*)[32]>(&r[32 * c]));
            tc_wait_ld();
            // The thread holds kOq columns of its own row; stored from here, every instruction of the warp would touch 32
            // different rows.  So the warp's 32 x (2 kOq)-byte block goes through the tile ring (free: the last product has
            // completed, and with it every read of the ring) and is written out with eight lanes per row - whole 128-byte
            // lines.  Rows padded by 16 bytes: the 16-byte accesses of eight lanes fall into different banks.
            constexpr int kRowB = C::kOq * 2, kPitch = kRowB + 16;          // bytes per row of the warp's block
            uint8_t *stg = smem + C::kRing + warp * (32 * kPitch);
#pragma unroll
            for (int j = 0; j < C::kOq / 8; ++j) {
                uint4 w;
                w.x = pack16<F16>(__uint_as_float(r[8 * j]) * inv, __uint_as_float(r[8 * j + 1]) * inv);
                w.y = pack16<F16>(__uint_as_float(r[8 * j + 2]) * inv, __uint_as_float(r[8 * j + 3]) * inv);
                w.z = pack16<F16>(__uint_as_float(r[8 * j + 4]) * inv, __uint_as_float(r[8 * j + 5]) * inv);
                w.w = pack16<F16>(__uint_as_float(r[8 * j + 6]) * inv, __uint_as_float(r[8 * j + 7]) * inv);
                *reinterpret_cast<uint4 *>(stg + lane * kPitch + 16 * j) = w;
            }
            __syncwarp();
            constexpr int kLanesPerRow = kRowB / 16, kRowsPerIt = 32 / kLanesPerRow;
            const int sub = lane / kLanesPerRow, ch = lane % kLanesPerRow;
            uint16_t *obase = p.out + b * p.o_sb + hq * p.o_sh + g * C::kOq + 8 * ch;
#pragma unroll
            for (int it = 0; it < 32 / kRowsPerIt; ++it) {
                const int rr = it * kRowsPerIt + sub;                           // row inside the warp's block
                const int64_t gr = static_cast<int64_t>(m) * kBlock + lq * 32 + rr;
                const uint4 w = *reinterpret_cast<const uint4 *>(stg + rr * kPitch + 16 * ch);
                if (gr < p.L) *reinterpret_cast<uint4 *>(obase + gr * p.o_sl) = w;
            }
            if (grow < p.L) {
                if (g == 0 && p.lse2) p.lse2[static_cast<int64_t>(bh) * p.L + grow] = ref + log2f(den);
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (s_err && tid == 0) {
        if (p.status) atomicExch(p.status, VQ_WORD_TIMEOUT);
        // a bounded wait expired: give tile loads still in flight time to land before leaving
#pragma unroll 1
        for (int w = 0; w < (1 << 14); ++w) __nanosleep(256);
    }
    __syncthreads();
    if (warp == C::kWarpTma) {
        __syncwarp();
        tmem_dealloc(tmem, C::kCols);
    }
}

template <int D, bool F16, int KEYS>
static int launch_tc4(const VqPrefillArgs *a, cudaStream_t stream)
{
    using C = T4Cfg<D, KEYS>;
    TcMaps m;
    TcParams p;
    const int st = tc_setup<D>(a, m, p, KEYS);
    if (st != VQ_OK) return st;
    auto kern = prefill_tc4_kernel<D, F16, KEYS>;
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, C::kTotal) != cudaSuccess ||
        cudaFuncSetAttribute(kern, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared) != cudaSuccess)
        return VQ_ELAUNCH;
    dim3 grid(static_cast<unsigned>(p.ntiles * (p.Hq / p.Hkv)), static_cast<unsigned>(a->q1.shape[0] * p.Hkv));
    kern<<<grid, C::kThreads, C::kTotal, stream>>>(m.q1, m.q2, m.k1, m.k3, m.v, m.cb, m.vs, p);
    return launch_status();
}

// 128-key steps cost less per key (one hand-off instead of two), two CTAs per SM cover each other's start and end, which weigh
// more the fewer items a tile has, and need more CTAs than SMs.  So the line lies at the mean number of items per tile.
// Measured: time of the 128-key form over that of the 64-key form, D = 128, L = 2048, 1184 CTAs: 1.25 at a mean of 4.4 items, 1.09
// at 7.1, 0.97 at 9.9 (ReRoPE, two passes over the boundary block: 1.02 at 10.6, 0.94 at 13.4), 0.83 at 18.8; D = 64, and 208 to
// 2048 CTAs, within 0.08 of that.  In us:
// 32768 tokens, 32 heads, MK1024, W1024: 1171 / 1244.  No more CTAs than SMs: 64 CTAs, 1024 tokens 17.5 / 25.2; 128 CTAs, 16384
// tokens, MK2048 37.0 / 63.2; 96 CTAs, 300 tokens 8.8 / 10.5; but one tile of one item 8.0 / 6.9.
template <int D, bool F16>
static int launch_keys(const VqPrefillArgs *a, cudaStream_t stream)
{
    int dev = 0, sms = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return VQ_EDEVICE;
    const int64_t tiles = (a->q1.shape[2] + kBlock - 1) / kBlock, ctas = a->q1.shape[0] * a->q1.shape[1] * tiles;
    const int64_t w = a->window / kBlock, past = tiles > w ? tiles - w : 0, in = tiles - past;   // tiles with and without a boundary block
    const bool far = a->codebook.ptr != nullptr && a->cnt.ptr != nullptr && past > 1, rerope = a->q2.ptr != a->q1.ptr || a->k3.ptr != a->k1.ptr;
    const int64_t items = in * (in + 1) / 2 + past * (w + (rerope ? 2 : 1)) + (far ? (past - 1) * (a->codebook.shape[1] / kBlock) : 0);
    const bool wide = ctas <= sms ? tiles > 1 : items >= (rerope ? 12 : 10) * tiles;
    return wide ? launch_tc4<D, F16, 128>(a, stream) : launch_tc4<D, F16, 64>(a, stream);
}

int launch_prefill_tensor4(const VqPrefillArgs *a, cudaStream_t stream)
{
    const int D = static_cast<int>(a->q1.shape[3]);
    // 16-byte aligned rows for the output stores and the tensor maps
    if (a->out.stride[2] % 8 || a->out.stride[1] % 8 || a->out.stride[0] % 8) return VQ_EINVAL_STRIDE;
    if (a->q1.dtype == VQ_F16) return D == 64 ? launch_keys<64, true>(a, stream) : launch_keys<128, true>(a, stream);
    return D == 64 ? launch_keys<64, false>(a, stream) : launch_keys<128, false>(a, stream);
}

}  // namespace vq
