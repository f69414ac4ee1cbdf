// Key -> code assignment with the score matrix on the tensor cores, still bit-exact.
//
// Replaces ops/mini_vq.py:4-18 of the reference (and its greedy-residual extension to M codebooks)
// for bf16, half and fp32 keys.  The defining arithmetic is unchanged: the code of a key in codebook m is the first
// arg-max over c of the fp32 fused-multiply-add chain  sum_d r_m[d] * C_m[c][d] (+ bias),
// r_0 = k, r_{m+1} = r_m - C_m[code] (fp32 subtraction).  What changes is how the arg-max is found:
//   1. APPROXIMATE scores of a 128-key tile against all K codewords come from tcgen05.mma.  The
//      fp32 codebook is split into two bf16 terms, C = Ch + Cl + eC with |eC| <= 2^-18 |C|.  The
//      residual is carried as two bf16 terms as well, rho_m = Rh + Rl (bf16 keys: rho_0 = k exactly, Rl = 0; half keys:
//      rho_0 = k exactly, 8 + 8 >= 11 significant bits; fp32 keys: |rho_0 - k| <= 2^-18 |k|, one more re-split);
//      after the code of codebook m is known, t = (Rh + Rl) - C_m[code] in fp32 is re-split.  The
//      tensor cores form  s~ = Rh.Ch + Rl.Ch + Rh.Cl  with fp32 accumulation.
//   2. Error of s~ against the defining chain, in units of |r| |C| (|r|: the norm of the residual,
//      bounded from the residual itself, which the thread has in hand when it re-splits it; a priori
//      |r| <= |k| + sum of the largest codeword norms of the codebooks before m):
//      split of C and dropped Rl.Cl: 2 * 2^-18;
//      re-splits of the residual: m * (2^-18 + 3 * 2^-24);  the fp32 chain itself: D * 2^-24 <= 2^-17;
//      tensor-core accumulation of 3 D (codebook 0: 2 D) exact products, each addition truncated to fp32:
//      3 D * 2^-23 <= 12 * 2^-18;  index tag in the low five mantissa bits (see tag_score): 2^-18.
//      Sum for D = 128: 13 units of 2^-18 for codebook 0, 17 + 1.05 m for codebook m; the kernel uses
//      eps_m = (4 + D/64 + (2 or 3) D/32 + 1.1 m) 2^-18, one unit above that; with keys that start as two terms (half,
//      fp32) codebook 0 has three products as well and every codebook one re-split more (1.1 (m + 1)).
//      A key whose best approximate score leads the runner-up by more than thr = 2 eps |r| max|C_m|
//      has a unique arg-max: that code is final.
//   3. The other keys (well under one per cent of the (key, codebook) pairs for random data) keep the
//      approximate winner for the time being.  Their candidates - the codes whose approximate score is
//      within thr of the best; the exact arg-max is among them - are written to a record (up to four codes;
//      more means "all of them"), the records of a key are chained, and the key
//      goes on a work list.  (A key of zeros ties with every finite code; its code is known without that.)  A second, small kernel (assign_repair_kernel) walks the list: it follows the
//      key through the codebooks with the defining fp32 arithmetic, runs the defining chain for the
//      candidates of every doubtful codebook (first maximum wins), and - in the rare case that this changes
//      a code - recomputes every later codebook of that key over all its codewords, since its residual
//      changed.  The scan kernel never waits for any of this.  Where too many keys have a whole codebook to score, the
//      second kernel scores all keys instead, in tiles that share the codebook (settle_all).
//      When a codebook is larger than the 256 score columns a stream owns in tensor memory (K = 512, 1024), its
//      chunks pass through that region in rounds and the scores of a chunk are gone once the next one lands.  The
//      candidates are then tracked during the scan: best, runner-up (each with its group of 32 codes) and the third
//      largest of all group maxima and group runners-up - and, for a group whose runner-up came within thr of the
//      running best, of the group's third score, looked up at once while it is there.  The cut only rises with the
//      running best, so a third below it excludes every other code: a group that was not looked up has its runner-up,
//      and with it its other 30 scores, below the cut.  Then the best and the runner-up are the only candidates;
//      otherwise, and always with a bias (thr then moves with the best score), the record says "all of them".
//      (Up to K = 384 the scores are still there: a group whose runner-up came near sets a flag, and such a key takes a
//      second look.)
// One CTA owns NS key tiles of 128 keys ("streams", NS = 2 except for K = 384): per stream eight warps,
// two threads per key, each ranking half of the key's scores in tensor memory and updating half of
// its residual row (the arithmetic between the MMAs is a chain of dependent instructions and loads
// from L2: it needs the warps to hide its latency); one warp issues the MMAs of the streams in turn,
// so the scan of one stream overlaps the MMAs of the other; one warp issues the TMA loads of the
// codebook terms (16 KB units, 5-slot ring).  Every wait is bounded.
// Half keys (B1 H32 D128 L5001, one codebook of 1024), all kernels: 164 us; on the exact kernel, which half and fp32 keys took
// before, 1440 us.
#include <type_traits>

#include "prefill_tc_common.cuh"

namespace vq {

using namespace ptx;

constexpr int kAtMinChunk = 128;   // codewords per MMA chunk: 128, or 256 (one N = 256 instruction) when K allows
constexpr int kAtMaxM = 8;
constexpr int kAtMaxK = 1024;   // 32 groups of 32 codes: one bit each in a thread's group mask
constexpr unsigned int kAtLeft = 64;
constexpr int kAtRepairWarps = 4;  // warps per CTA of the repair kernel (one doubtful key per warp at a time)

// ------------------------------------------------------------------------------------------------
// fp32 codebook -> bf16 hi / lo terms [Hkv, M*K, D], the squared norm of every row and the largest row
// norm of every codebook (grid.x: codebook, grid.y: slices of kSplitRows rows; cmax zeroed by the launcher, the
// slices meet in it through an atomic maximum on the bits of their non-negative norms).
constexpr int kSplitRows = 64;   // divides kAtMinChunk, of which every K here is a multiple
// Floor of the squared norms that error bounds are formed from: the squares of elements below 1e-22 vanish in fp32, and a
// bound of zero would declare every lead safe.
constexpr float kAtMinNorm2 = 1e-35f;
template <int D>
__global__ void __launch_bounds__(256)
split_codebook_kernel(const float *__restrict__ cb, __nv_bfloat16 *__restrict__ hi, __nv_bfloat16 *__restrict__ lo,
                      float *__restrict__ cmax, float *__restrict__ cn2, unsigned int *__restrict__ work_count, int K)
{
    // D/4 lanes to a row, four columns a lane; a warp's rows are all in flight together (16 MB of codebooks, 32 heads x 4 x 256:
    // 11.9 -> 8.0 us against one column per lane and load, one row at a time)
    constexpr int LPR = D / 4, RPI = 32 / LPR, NIT = kSplitRows / 8 / RPI;   // lanes per row, rows per instruction, instructions
    __shared__ float s_max[8];
    if (blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x < 3) work_count[threadIdx.x] = 0u;   // the scan kernel that follows fills the lists
    const int hm = blockIdx.x;  // h * M + m
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int c0 = static_cast<int>(blockIdx.y) * kSplitRows + warp * (kSplitRows / 8) + lane / LPR;   // K is a multiple of kSplitRows
    const int64_t base = (static_cast<int64_t>(hm) * K + c0) * D + 4 * (lane % LPR);
    float4 x[NIT];
#pragma unroll
    for (int i = 0; i < NIT; ++i) x[i] = __ldg(reinterpret_cast<const float4 *>(cb + base + static_cast<int64_t>(i) * RPI * D));
    float wmax = 0.f;
#pragma unroll
    for (int i = 0; i < NIT; ++i) {
        const float v[4] = {x[i].x, x[i].y, x[i].z, x[i].w};
        uint32_t wh[2], wl[2];
        float ss = 0.f;
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            wh[e] = pack_bf16(v[2 * e], v[2 * e + 1]);
            wl[e] = pack_bf16(v[2 * e] - __uint_as_float(wh[e] << 16), v[2 * e + 1] - __uint_as_float(wh[e] & 0xffff0000u));
            ss = fmaf(v[2 * e], v[2 * e], fmaf(v[2 * e + 1], v[2 * e + 1], ss));
        }
        *reinterpret_cast<uint2 *>(hi + base + static_cast<int64_t>(i) * RPI * D) = make_uint2(wh[0], wh[1]);
        *reinterpret_cast<uint2 *>(lo + base + static_cast<int64_t>(i) * RPI * D) = make_uint2(wl[0], wl[1]);
#pragma unroll
        for (int off = LPR / 2; off >= 1; off >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, off);
        if (lane % LPR == 0) cn2[static_cast<int64_t>(hm) * K + c0 + i * RPI] = ss;
        wmax = fmaxf(wmax, sqrtf(fmaxf(ss, kAtMinNorm2)));
    }
    if (RPI > 1) wmax = fmaxf(wmax, __shfl_xor_sync(0xffffffffu, wmax, 16));
    if (lane == 0) s_max[warp] = wmax;
    __syncthreads();
    if (threadIdx.x == 0) {
        float m = 0.f;
        for (int w = 0; w < 8; ++w) m = fmaxf(m, s_max[w]);
        atomicMax(reinterpret_cast<unsigned int *>(cmax + hm), __float_as_uint(m * 1.0001f));  // sqrt / summation rounding
    }
}

struct AtParams {
    const void *k;       // bf16, half or fp32 rows
    int64_t k_sb, k_sh, k_sl;
    const float *cb;     // [Hkv, M, K, D]
    const float *bias;   // nullptr or [Hkv, M, K]
    const float *cmax;   // [Hkv, M]
    const float *cn2;    // [Hkv, M*K] squared row norms
    void *codes;
    int code_dtype;
    int64_t c_sb, c_sh, c_sl;
    int Hkv, M, K, ntiles;
    int64_t L;
    int32_t *status;
    long long wait_limit;  // cycles a device-side wait may last before the kernel gives up
    uint4 *work;                // doubtful keys: {key index lo, hi, last record, doubtful codebooks | brute-force codebooks << 8};
                                // from the front those whose candidates are known, from the back the others (one entry per key in all)
    uint4 *pool;                // candidate records: {previous record of the key, m | n << 8, codes 0-1, codes 2-3}
    unsigned int *counters;     // [0] entries at the front of `work`, [1] records in `pool`, [2] entries at the back (zeroed by split_codebook_kernel)
    unsigned int pool_cap;      // records in `pool` and entries in `work`: one per key
};

template <int D, int NS, int CH>
struct AtCfg {
    static constexpr int NH = D / 64;
    static constexpr int kATile = NH * kHalfBytes;     // 128 keys x D bf16 (one term of the residual)
    static constexpr int kUnit = CH * 64 * 2;          // CH codewords x 64 columns of one term: one ring slot
    static constexpr int kSlots = 80 * 1024 / kUnit;   // 80 KB of ring
    static constexpr int kB = NS * 2 * kATile;         // per stream: Rh then Rl
    static constexpr int kTotal = kB + kSlots * kUnit + 1024;
    static constexpr int kRegion = NS == 2 ? 256 : 512;  // score columns of a stream in tensor memory
    static constexpr int kMaxChunks = kRegion / CH;
    static constexpr int kGroupsPerChunk = CH / 32;
    static constexpr int kMaxGroups = kRegion / 32;
    static constexpr int kScanWarps = 8;               // per stream: two threads per key
    static constexpr int kWarpMma = kScanWarps * NS, kWarpTma = kScanWarps * NS + 1;
    static constexpr int kThreads = (kScanWarps * NS + 2) * 32;
};

// Largest (hi) and second largest (lo) of 32 values: pairs, then merges of (hi, lo) pairs.
__device__ __forceinline__ void top2_32(const float (&v)[32], float &hi, float &lo)
{
    float h[16], l[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) {
        h[i] = fmaxf(v[2 * i], v[2 * i + 1]);
        l[i] = fminf(v[2 * i], v[2 * i + 1]);
    }
#pragma unroll
    for (int n = 8; n >= 1; n >>= 1)
#pragma unroll
        for (int i = 0; i < n; ++i) {
            const float a = h[2 * i], b = h[2 * i + 1];
            l[i] = fmax3(fminf(a, b), l[2 * i], l[2 * i + 1]);
            h[i] = fmaxf(a, b);
        }
    hi = h[0];
    lo = l[0];
}

// A score with its low five mantissa bits replaced by 31 - i (i: index inside a group of 32 codes):
// the maximum of such values carries the index of a maximal element; the values move by < 2^-18 |v|.
__device__ __forceinline__ float tag_score(float v, int i)
{
    return __uint_as_float((__float_as_uint(v) & 0xffffffe0u) | static_cast<uint32_t>(31 - i));
}

// 32 score columns of this thread's key as floats (+ bias of their codes)
__device__ __forceinline__ void load_scores(uint32_t taddr, const float *bm, int c0, float (&v)[32])
{
    uint32_t r[32];
    tmem_ld32(taddr, r);
    tc_wait_ld();
#pragma unroll
    for (int i = 0; i < 32; ++i) v[i] = __uint_as_float(r[i]);
    // one branch over all of it: tested per element, the loads and additions are issued predicated off (a seventh of the
    // kernel's instructions)
    if (bm != nullptr) {
#pragma unroll
        for (int i = 0; i < 32; ++i) v[i] += __ldg(bm + c0 + i);
    }
}

__device__ __forceinline__ void st_shared8(uint32_t addr, uint32_t x, uint32_t y) { asm volatile("st.shared.v2.u32 [%0], {%1, %2};" ::"r"(addr), "r"(x), "r"(y) : "memory"); }
__device__ __forceinline__ uint2 ld_shared8(uint32_t addr)
{
    uint2 v;
    asm volatile("ld.shared.v2.u32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "r"(addr) : "memory");
    return v;
}

// four residual columns as bf16 hi and lo terms, 8 bytes each, at byte `off` of the two operand tiles (packed conversions:
// single ones run on the special-function unit, a quarter of the rate)
__device__ __forceinline__ void store_terms(uint32_t a_rh, uint32_t a_rl, uint32_t off, const float (&x)[4])   // shared-memory addresses
{
    uint32_t wh[2], wl[2];
#pragma unroll
    for (int e = 0; e < 2; ++e) {
        wh[e] = pack_bf16(x[2 * e], x[2 * e + 1]);
        float l0, l1;   // x - hi
        ffma2(l0, l1, __uint_as_float(wh[e] << 16), __uint_as_float(wh[e] & 0xffff0000u), -1.f, -1.f, x[2 * e], x[2 * e + 1]);
        wl[e] = pack_bf16(l0, l1);
    }
    st_shared8(a_rh + off, wh[0], wh[1]);
    st_shared8(a_rl + off, wl[0], wl[1]);
}

// WRAP: a codebook has more chunks than the stream's score region holds and goes through it in rounds.
// KT: key type.  bf16 keys are the first residual as they lie in memory (a TMA tile); half and fp32 keys are split into two
// bf16 terms by the scan warps first (kConv).
template <typename KT, int D, int NS, int CH, bool WRAP>
__global__ void __launch_bounds__(AtCfg<D, NS, CH>::kThreads, 1)
assign_tc_kernel(const __grid_constant__ CUtensorMap tm_k, const __grid_constant__ CUtensorMap tm_hi,
                 const __grid_constant__ CUtensorMap tm_lo, AtParams p)
{
    using C = AtCfg<D, NS, CH>;
    constexpr int NH = C::NH, SL = C::kSlots;
    constexpr bool kConv = !std::is_same<KT, __nv_bfloat16>::value;
    extern __shared__ uint8_t smem_raw[];
    uint8_t *smem = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    __shared__ __align__(8) uint64_t bar_k[NS], bar_q[NS], bar_c[NS][C::kMaxChunks], c_free[NS][C::kMaxChunks], b_full[SL], b_free[SL];
    __shared__ __align__(8) uint64_t x_half[NS][4], x_done[NS][4];   // hand-offs between the two warps of a lane quarter
    __shared__ __align__(16) float4 s_x[NS][kBlock];                  // per key: what its two threads tell each other
    __shared__ __align__(16) float4 s_y[NS][kBlock];                  // ... the rest of it (third best, runner-up's group, flag)
    __shared__ float s_norm2[kConv ? NS : 1][kConv ? kBlock : 1];     // squared norms of the keys that the scan warps split
    __shared__ uint32_t s_tmem;
    __shared__ int s_err;

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int u = blockIdx.y, b = u / p.Hkv, h = u % p.Hkv;
    const int M = p.M, K = p.K, MK = M * K;
    const int chunks = K / CH;
    // A codebook with more chunks than the stream's score region holds (K = 1024: four chunks of 256 columns in a region of
    // 512) goes through the region in rounds: chunk ch lands in slot ch mod kMaxChunks once the scan threads have
    // released the chunk that was there; `rounds` uses of every slot per codebook.
    constexpr bool wrap = WRAP;                        // (the launcher picks WRAP = chunks > kMaxChunks)
    const int rounds = wrap ? chunks / C::kMaxChunks : 1;
    const int tile0 = static_cast<int>(blockIdx.x) * NS;
    const int n_act = min(NS, p.ntiles - tile0);       // streams with a tile

    if (tid == 0) {
        for (int i = 0; i < NS; ++i) {
            mbar_init(&bar_k[i], 1);
            mbar_init(&bar_q[i], 32 * C::kScanWarps);
            for (int qd = 0; qd < 4; ++qd) {
                mbar_init(&x_half[i][qd], 1);
                mbar_init(&x_done[i][qd], 1);
            }
            for (int c = 0; c < C::kMaxChunks; ++c) {
                mbar_init(&bar_c[i][c], 1);
                mbar_init(&c_free[i][c], C::kScanWarps);
            }
        }
        for (int i = 0; i < SL; ++i) {
            mbar_init(&b_full[i], 1);
            mbar_init(&b_free[i], 1);
        }
        fence_mbar_init();
        s_err = 0;
    }
    if (warp == C::kWarpMma) {
        __syncwarp();
        tmem_alloc(&s_tmem, 512u);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = s_tmem;

    if (warp == C::kWarpTma) {
        // ============================================================ TMA producer
        if (elect_one()) {
            if (!kConv) prefetch_tmap(&tm_k);
            prefetch_tmap(&tm_hi); prefetch_tmap(&tm_lo);
            for (int s = 0; s < n_act && !kConv; ++s) {
                mbar_expect_tx(&bar_k[s], C::kATile);
#pragma unroll
                for (int hh = 0; hh < NH; ++hh)
                    tma_load_4d(smem + s * 2 * C::kATile + hh * kHalfBytes, &tm_k, &bar_k[s], 64 * hh, (tile0 + s) * kBlock, h, b);
            }
            // Units in the order the MMA warp consumes them: per codebook m the chunks in turn, each chunk for the
            // streams in turn (so that the scan of one stream's chunk runs under the other stream's MMAs); per
            // (chunk, stream): hi term columns 0-63, 64-127 (D = 128), then the lo term likewise.
            // (nested counters instead of divisions of a flat index: this thread's instructions are serial)
            bool ok = true;
            int g = 0;
            for (int m = 0; m < M && ok; ++m)
                for (int ch = 0; ch < chunks && ok; ++ch)
                    for (int s = 0; s < n_act && ok; ++s)
#pragma unroll
                        for (int rem = 0; rem < 2 * NH; ++rem, ++g) {
                            const int slot = g % SL, is_lo = rem / NH, hh = rem % NH;
                            if (g >= SL && !mbar_wait(&b_free[slot], ((g / SL) - 1) & 1, p.wait_limit)) {
                                ok = false;
                                break;
                            }
                            const int row = h * MK + m * K + ch * CH;  // row in [Hkv*M*K, D]
                            mbar_expect_tx(&b_full[slot], C::kUnit);
                            tma_load_3d(smem + C::kB + slot * C::kUnit, is_lo ? &tm_lo : &tm_hi, &b_full[slot], 64 * hh, row, 0);
                        }
            if (!ok) s_err = 1;
        }
    } else if (warp == C::kWarpMma) {
        // ============================================================ MMA issuer
        if (elect_one()) {
            constexpr uint32_t idesc = idesc_bf16(128, CH, 0, 0, 0);
            // descriptors differ only in their 16-byte-granular start address: build the bases once
            const uint64_t d_a0 = smem_desc_sw128(smem_u32(smem), 16, 1024);
            const uint64_t d_b0 = smem_desc_sw128(smem_u32(smem + C::kB), 16, 1024);
            bool ok = true;
            int g = 0;
            for (int m = 0; m < M && ok; ++m)
                for (int ch = 0; ch < chunks && ok; ++ch)
                    for (int s = 0; s < n_act && ok; ++s) {
                        // the residual terms of (s, m): a bf16 key tile itself for m = 0, else written by the scan threads
                        if (ch == 0 && !(m == 0 && !kConv ? mbar_wait(&bar_k[s], 0, p.wait_limit)
                                                          : mbar_wait(&bar_q[s], (kConv ? m : m - 1) & 1, p.wait_limit))) {
                            ok = false;
                            break;
                        }
                        const int cs = wrap ? ch % C::kMaxChunks : ch, use = m * rounds + (wrap ? ch / C::kMaxChunks : 0);
                        if (wrap && use >= 1 && !mbar_wait(&c_free[s][cs], (use - 1) & 1, p.wait_limit)) {   // the slot's previous chunk has been scanned
                            ok = false;
                            break;
                        }
                        if (ch == 0 || wrap) tc_fence_after();
                        const uint32_t dcol = tmem + s * C::kRegion + cs * CH;
#pragma unroll
                        for (int rem = 0; rem < 2 * NH; ++rem, ++g) {
                            const int slot = g % SL, is_lo = rem / NH, hh = rem % NH;
                            if (!mbar_wait(&b_full[slot], (g / SL) & 1, p.wait_limit)) {
                                ok = false;
                                break;
                            }
                            tc_fence_after();
                            const uint64_t d_b = d_b0 + static_cast<uint64_t>((slot * C::kUnit) >> 4);
                            const uint64_t d_rh = d_a0 + static_cast<uint64_t>((s * 2 * C::kATile + hh * kHalfBytes) >> 4);
                            const uint64_t d_rl = d_rh + static_cast<uint64_t>(C::kATile >> 4);
#pragma unroll
                            for (int k4 = 0; k4 < 4; ++k4)
                                mma_ss(dcol, d_rh + static_cast<uint64_t>((k4 * 32) >> 4), d_b + static_cast<uint64_t>((k4 * 32) >> 4), idesc,
                                       (rem | k4) ? 1u : 0u);
                            if (!is_lo && (kConv || m > 0)) {
#pragma unroll
                                for (int k4 = 0; k4 < 4; ++k4)
                                    mma_ss(dcol, d_rl + static_cast<uint64_t>((k4 * 32) >> 4), d_b + static_cast<uint64_t>((k4 * 32) >> 4), idesc, 1u);
                            }
                            tc_commit(&b_free[slot]);
                            if (rem == 2 * NH - 1) tc_commit(&bar_c[s][cs]);  // this chunk's score columns are complete
                        }
                    }
            if (!ok) s_err = 1;
        }
    } else if (warp / C::kScanWarps < n_act) {
        // ============================================================ scan warps: two threads per key
        // Thread (hf, row) ranks the groups [hf * groups / 2, (hf + 1) * groups / 2) of its key's scores and
        // updates half hf of its residual row; the two meet through shared memory once per codebook.
        constexpr unsigned kAll = 0xffffffffu;
        const int s = warp / C::kScanWarps, hf = (warp >> 2) & 1, wq = warp & 3;
        const int row = wq * 32 + lane;
        const int64_t j0 = static_cast<int64_t>(tile0 + s) * kBlock;
        const int64_t j = j0 + row;
        const bool valid = j < p.L;
        const uint32_t tbase = tmem + (static_cast<uint32_t>(wq * 32) << 16) + s * C::kRegion;
        const float *cbh = p.cb + static_cast<int64_t>(h) * MK * D;
        uint8_t *a_tile = smem + s * 2 * C::kATile;
        const uint32_t a_rh = smem_u32(a_tile), a_rl = a_rh + C::kATile;
        const int groups = K / 32, g_lo = hf * (groups / 2), g_hi = g_lo + groups / 2;
        float4 *xch = &s_x[s][row];
        float rbound;  // |k| + sum of the largest codeword norms so far: a priori bound of the residual's norm
        float rnow;    // bound of the current residual's norm (tighter): see the residual update below
        bool zero_key;  // every element is zero (padding): see `tied` below
        bool ok = true;
        if constexpr (kConv) {
            // ---- the keys of this stream as two bf16 terms in the operand layout, and their squared norms.  As in the
            // residual update below a warp walks 16 of its quarter's keys, D/4 lanes per key: whole rows per load.
            constexpr int LPR = D / 4, KPI = 32 / LPR, NIT = 16 / KPI;
            const int sub = lane / LPR, l = lane % LPR;
            const uint32_t lane_off = (l >> 4) * kHalfBytes + 8 * (l & 1);
            const int chunk = (l & 15) >> 1;
            const KT *kb = static_cast<const KT *>(p.k) + b * p.k_sb + h * p.k_sh + 4 * l;
#pragma unroll 4
            for (int i = 0; i < NIT; ++i) {
                const int r = wq * 32 + 16 * hf + i * KPI + sub;
                float x[4] = {0.f, 0.f, 0.f, 0.f};
                if (j0 + r < p.L) {
                    if constexpr (std::is_same<KT, float>::value) {
                        const float4 v = __ldg(reinterpret_cast<const float4 *>(kb + (j0 + r) * p.k_sl));
                        x[0] = v.x; x[1] = v.y; x[2] = v.z; x[3] = v.w;
                    } else {
                        const uint2 v = __ldg(reinterpret_cast<const uint2 *>(kb + (j0 + r) * p.k_sl));
                        const float2 f0 = Pair16<KT>::unpack(v.x), f1 = Pair16<KT>::unpack(v.y);
                        x[0] = f0.x; x[1] = f0.y; x[2] = f1.x; x[3] = f1.y;
                    }
                }
                store_terms(a_rh, a_rl, lane_off + r * 128 + ((chunk ^ (r & 7)) << 4), x);
                float ss = fmaf(x[0], x[0], fmaf(x[1], x[1], fmaf(x[2], x[2], x[3] * x[3])));
                if constexpr (std::is_same<KT, float>::value)   // where only the squares vanish: not zero
                    ss += fminf(fmaxf(fmaxf(fabsf(x[0]), fabsf(x[1])), fmaxf(fabsf(x[2]), fabsf(x[3]))), 1e-44f);
#pragma unroll
                for (int off = LPR / 2; off >= 1; off >>= 1) ss += __shfl_xor_sync(kAll, ss, off);
                if (l == 0) s_norm2[s][r] = ss;
            }
            fence_proxy_async_smem();
            mbar_arrive(&bar_q[s]);
            ok = __all_sync(kAll, mbar_wait(&bar_q[s], 0, p.wait_limit));   // every warp's part, this row's norm among them
            rbound = sqrtf(fmaxf(s_norm2[s][row], kAtMinNorm2)) * 1.0001f;
            zero_key = s_norm2[s][row] == 0.f;
            rnow = rbound;
        } else {
            ok = __all_sync(kAll, mbar_wait(&bar_k[s], 0, p.wait_limit));
            // |k| from the key tile the TMA load put into shared memory (this thread's row, 16-byte chunks in the
            // 128-byte swizzle: eight consecutive rows read eight different chunks, so the reads do not collide)
            float ss = 0.f;
            uint32_t any = 0;
#pragma unroll 4
            for (int ck = 0; ck < D / 8; ++ck) {
                const uint4 raw = *reinterpret_cast<const uint4 *>(a_tile + (ck >> 3) * kHalfBytes + row * 128 + (((ck & 7) ^ (row & 7)) << 4));
                any |= raw.x | raw.y | raw.z | raw.w;
                const __nv_bfloat162 *hp = reinterpret_cast<const __nv_bfloat162 *>(&raw);
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const float x = __low2float(hp[i]), y = __high2float(hp[i]);
                    ss = fmaf(x, x, fmaf(y, y, ss));
                }
            }
            rbound = sqrtf(fmaxf(ss, kAtMinNorm2)) * 1.0001f;
            rnow = rbound;
            zero_key = (any & 0x7fff7fffu) == 0u;
        }
        uint32_t doubt = 0;   // bit m: the lead of codebook m's best score did not prove its arg-max (bit 8 + m: no record)
        uint32_t last_rec = 0xffffffffu;   // the key's most recent candidate record
        bool heavy = false;                // a whole codebook has to be scored
        for (int m = 0; m < M && ok; ++m) {
            const float cm = p.cmax[h * M + m];
            // eps of this codebook in units of 2^-18: the terms listed at the top of the file plus one unit of slack
            const int splits = kConv ? m + 1 : m;   // re-splits that the residual has been through
            const float eps_m = (4.f + D / 64 + (splits > 0 ? 3 : 2) * (D / 32) + 1.1f * splits) * 3.814697265625e-6f;
            const float thr0 = 2.f * eps_m * rnow * cm + 1e-30f;
            const float *bm = p.bias ? p.bias + (static_cast<int64_t>(h) * M + m) * K : nullptr;
            // A key of zeros scores +0 with every code whose entries are finite (NaN with the others): without a bias the
            // first code is its arg-max if that code is finite, and no lead has to prove it.
            const bool tied = m == 0 && zero_key && bm == nullptr && __ldg(p.cn2 + static_cast<int64_t>(h) * MK) < INFINITY;
            // ---- scan of this thread's groups, chunk by chunk as the tensor pipe finishes them: best and runner-up
            // of the tagged scores (the tag of the best gives its index inside its group of 32)
            float best = -INFINITY, second = -INFINITY;
            int bgrp = g_lo;
            uint32_t gbits = 0;   // groups whose maximum came within the threshold of the running best: a superset of
                                  // the groups that can hold a candidate at the end
            // The candidates of a key that turns out doubtful are tracked on the way: the group of the runner-up, the third
            // largest of all group maxima and group runners-up, and whether the runner-up of any group came within the
            // threshold of the running best (the other 30 scores of such a group are unknown here and may hold further
            // candidates).  A doubtful key whose third lies below the cut needs no second look at its scores - which WRAP
            // could not take anyway: the scores of earlier chunks are gone by then, so there the third of such a group is
            // looked up at once (M4 K512, 2 x 16384 tokens x 32 heads: 279 -> 115 us of repair beside 1.38 ms of scan).
            float third = -INFINITY;
            int sgrp = g_lo;
            bool amb = bm != nullptr;   // with a bias the threshold moves with the best score: no short list then
            auto rank_group = [&](int g, uint32_t col) {   // group g of the codebook, its 32 score columns at `col` of the stream's region
                float v[32];
                load_scores(tbase + col, bm, 32 * g, v);
#pragma unroll
                for (int i = 0; i < 32; ++i) v[i] = tag_score(v[i], i);
                float hi, lo;
                top2_32(v, hi, lo);
                // hi, then lo (<= hi) into the sorted triple (best, second, third); a tie with the best goes to the
                // earlier group, which holds the lower codes
                // (minima, maxima and selects: as branches the lanes of a warp take different ones)
                const bool new_best = hi > best;
                const float beaten = fminf(hi, best), s1 = fmaxf(second, beaten);
                sgrp = new_best ? bgrp : hi > second ? g : sgrp;
                sgrp = lo > s1 ? g : sgrp;
                bgrp = new_best ? g : bgrp;
                third = fmax3(third, fminf(second, beaten), fminf(s1, lo));
                second = fmaxf(s1, lo);
                best = fmaxf(best, hi);
                if constexpr (wrap) {
                    // a group whose runner-up came near gives up its third as well: there is no second look later
                    const bool near_best = valid && !tied && lo >= best - thr0;   // (rows past the end are zeros as well)
                    if (__any_sync(kAll, near_best)) {
                        load_scores(tbase + col, bm, 32 * g, v);
                        float g3 = -INFINITY;
#pragma unroll
                        for (int i = 0; i < 32; ++i) {
                            const float x = tag_score(v[i], i);   // (the tags make the 32 values distinct)
                            g3 = fmaxf(g3, x == hi || x == lo ? -INFINITY : x);
                        }
                        if (near_best) third = fmaxf(third, g3);
                    }
                } else {
                    amb |= lo >= best - thr0;
                }
                if constexpr (!wrap) {
                    // for the keys that do need a second look: the groups whose maximum came within the threshold
                    // (with a bias the fp32 additions s + bias round by up to 2^-24 |s + bias| each)
                    const float thr_g = bm ? thr0 + fabsf(best) * 4.76837158203125e-7f : thr0;
                    gbits |= (hi >= best - thr_g ? 1u : 0u) << g;
                }
            };
            if constexpr (!wrap) {
#pragma unroll 1
                for (int g = g_lo; g < g_hi && ok; ++g) {
                    if (g == g_lo || g % C::kGroupsPerChunk == 0) {
                        ok = __all_sync(kAll, mbar_wait(&bar_c[s][g / C::kGroupsPerChunk], m & 1, p.wait_limit));
                        tc_fence_after();
                        if (!ok) break;
                    }
                    rank_group(g, 32 * g);
                }
            } else {
                // rounds through the region: of every chunk this thread ranks half hf of the groups, then releases the slot
                constexpr int GPC = C::kGroupsPerChunk;
                bgrp = sgrp = hf * (GPC / 2);
#pragma unroll 1
                for (int ch = 0; ch < chunks && ok; ++ch) {
                    const int cs = ch % C::kMaxChunks, use = m * rounds + ch / C::kMaxChunks;
                    ok = __all_sync(kAll, mbar_wait(&bar_c[s][cs], use & 1, p.wait_limit));
                    tc_fence_after();
                    if (!ok) break;
#pragma unroll 1
                    for (int i = hf * (GPC / 2); i < (hf + 1) * (GPC / 2); ++i) rank_group(ch * GPC + i, cs * CH + 32 * i);
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&c_free[s][cs]);
                }
            }
            if (!ok) break;
            // ---- the two halves meet: the upper half hands its result over, the lower half merges (a tie between
            // the halves goes to the lower one, which holds the lower codes) and hands the result back
            int code;
            if (hf == 1) {
                *xch = make_float4(best, second, __int_as_float(bgrp), __uint_as_float(gbits));
                s_y[s][row] = make_float4(third, __int_as_float(sgrp), amb ? 1.f : 0.f, 0.f);
                __syncwarp();
                if (lane == 0) mbar_arrive(&x_half[s][wq]);
                ok = __all_sync(kAll, mbar_wait(&x_done[s][wq], m & 1, p.wait_limit));
                if (!ok) break;
                const float4 r = *xch;
                best = r.x;
                code = __float_as_int(r.y);
            } else {
                ok = __all_sync(kAll, mbar_wait(&x_half[s][wq], m & 1, p.wait_limit));
                if (!ok) break;
                const float4 o = *xch;
                {
                    // the other half's sorted triple into this one (its best with its group, its runner-up with its group, its third)
                    const float4 oy = s_y[s][row];
                    const int obg = __float_as_int(o.z), osg = __float_as_int(oy.y);
                    amb |= oy.z != 0.f;
                    if (o.x > best || (o.x == best && obg < bgrp)) {   // equal tagged scores: the lower group holds the lower code
                        third = second; second = best; sgrp = bgrp; best = o.x; bgrp = obg;
                    } else if (o.x > second) {
                        third = second; second = o.x; sgrp = obg;
                    } else {
                        third = fmaxf(third, o.x);
                    }
                    if (o.y > second) {
                        third = second; second = o.y; sgrp = osg;
                    } else {
                        third = fmaxf(third, o.y);
                    }
                    third = fmaxf(third, oy.x);
                }
                code = bgrp * 32 + 31 - static_cast<int>(__float_as_uint(best) & 31u);  // first group holding the maximum
                if (tied) code = 0;
                *xch = make_float4(best, __int_as_float(code), 0.f, 0.f);
                __syncwarp();
                if (lane == 0) mbar_arrive(&x_done[s][wq]);
                // with a bias the fp32 additions s + bias round by up to 2^-24 |s + bias| each
                const float thr = bm ? thr0 + fabsf(best) * 4.76837158203125e-7f : thr0;
                const bool dflag = valid && !tied && !(best - second > thr);
                if (__ballot_sync(kAll, dflag)) {
                    // ---- some key of this warp is doubtful: its candidates (scores within thr of the best) go into a
                    // record for the repair kernel; carry on with the approximate winner.  The best and the runner-up are
                    // the only candidates when the third largest tracked score is below the cut (and, where the third of a close
                    // group was not looked up, no group's runner-up came near the best).  The other doubtful keys take a second look at their scores (tensor-memory
                    // loads are warp-wide, so the warp re-reads the union of those keys' marked groups) - or, with WRAP,
                    // name every code a candidate (the repair kernel then scores the whole codebook).
                    const float cut = best - thr;
                    const bool quick = dflag && !amb && third < cut;
                    const bool slow = dflag && !quick;
                    int n = 0;
                    uint32_t c01 = 0, c23 = 0;
                    if (quick) {
                        n = 2;
                        c01 = static_cast<uint32_t>(code) |
                              (static_cast<uint32_t>(sgrp * 32 + 31 - static_cast<int>(__float_as_uint(second) & 31u)) << 16);
                    }
                    if (wrap && slow) n = 255;
                    const bool unbounded = !(thr < 3e38f);   // infinities, NaN or an overflowed norm: the approximate scores say nothing
                    const uint32_t gb = (!wrap && slow) ? (gbits | __float_as_uint(o.w)) : 0u;
                    const uint32_t un = __reduce_or_sync(kAll, gb);
#pragma unroll 1
                    for (int g = 0; g < groups && !wrap; ++g) {
                        if (!((un >> g) & 1u)) continue;
                        if (!__all_sync(kAll, mbar_wait(&bar_c[s][g / C::kGroupsPerChunk], m & 1, p.wait_limit))) {
                            ok = false;
                            break;
                        }
                        tc_fence_after();
                        float v[32];
                        load_scores(tbase + 32 * g, bm, 32 * g, v);
                        if ((gb >> g) & 1u) {
#pragma unroll
                            for (int i = 0; i < 32; ++i)
                                if (v[i] >= cut) {
                                    const uint32_t c = static_cast<uint32_t>(g * 32 + i);
                                    if (n < 2) c01 |= c << (16 * n);
                                    else if (n < 4) c23 |= c << (16 * (n - 2));
                                    ++n;
                                }
                        }
                    }
                    if (!ok) break;
                    if (dflag) {
                        const unsigned int at = atomicAdd(p.counters + 1, 1u);
                        if (at < p.pool_cap) {
                            if (unbounded || n > 4) n = 255;
                            heavy |= n == 255 || n == 0;
                            p.pool[at] = make_uint4(last_rec, static_cast<uint32_t>(m) | (static_cast<uint32_t>(n) << 8), c01, c23);
                            last_rec = at;
                            doubt |= 1u << m;
                        } else {
                            heavy = true;
                            doubt |= 0x100u << m;   // no room for the record: the repair kernel scores every code of this codebook
                        }
                    }
                }
                if (valid) store_code(p.codes, p.code_dtype, b * p.c_sb + h * p.c_sh + j * p.c_sl + m, code);
            }
            rbound += cm;
            if (m + 1 < M) {
                // ---- residual -= C_m[code] (fp32), re-split into bf16 hi / lo in the 128B-swizzled operand layout
                {
                    // The warp walks 16 of its quarter's 32 keys (the partner warp the other 16); D/4 lanes share a key, lane l
                    // of them owns its columns 4l .. 4l+3.  One load instruction then covers whole codebook rows - full
                    // 128-byte lines - where a thread fetching its own key's half row touched 32 different lines per
                    // instruction; eight loads are in flight at a time.
                    constexpr int LPR = D / 4, KPI = 32 / LPR, NIT = 16 / KPI;   // lanes per row, keys per instruction, instructions
                    constexpr int NB = NIT < 8 ? NIT : 8;                       // loads in flight (registers)
                    const int sub = lane / LPR, l = lane % LPR;
                    const uint32_t lane_off = (l >> 4) * kHalfBytes + 8 * (l & 1);   // the 64-column half and the 8 bytes inside a 16-byte chunk
                    const int chunk = (l & 15) >> 1;
#pragma unroll 1
                    for (int i0 = 0; i0 < NIT; i0 += NB) {
                        float4 crow4[NB];
#pragma unroll
                        for (int i = 0; i < NB; ++i) {
                            const int ck = __shfl_sync(kAll, code, 16 * hf + (i0 + i) * KPI + sub);
                            crow4[i] = __ldg(reinterpret_cast<const float4 *>(cbh + (static_cast<int64_t>(m) * K + ck) * D) + l);
                        }
#pragma unroll
                        for (int i = 0; i < NB; ++i) {
                            const int r = wq * 32 + 16 * hf + (i0 + i) * KPI + sub;
                            const uint32_t off = lane_off + r * 128 + ((chunk ^ (r & 7)) << 4);
                            const uint2 vh = ld_shared8(a_rh + off);
                            float x[4] = {__uint_as_float(vh.x << 16), __uint_as_float(vh.x & 0xffff0000u), __uint_as_float(vh.y << 16),
                                          __uint_as_float(vh.y & 0xffff0000u)};
                            if (kConv || m > 0) {
                                const uint2 vl = ld_shared8(a_rl + off);
                                fadd2(x[0], x[1], x[0], x[1], __uint_as_float(vl.x << 16), __uint_as_float(vl.x & 0xffff0000u));
                                fadd2(x[2], x[3], x[2], x[3], __uint_as_float(vl.y << 16), __uint_as_float(vl.y & 0xffff0000u));
                            }
                            ffma2(x[0], x[1], crow4[i].x, crow4[i].y, -1.f, -1.f, x[0], x[1]);
                            ffma2(x[2], x[3], crow4[i].z, crow4[i].w, -1.f, -1.f, x[2], x[3]);
                            store_terms(a_rh, a_rl, off, x);
                        }
                    }
                }
                // Norm of the new residual rho' = rho - C[code] without another pass over it:
                //   |rho'|^2 = |rho|^2 - 2 rho.C + |C|^2,   rho.C >= s - eps |rho| max|C|
                // where s is the tensor-core score the code was chosen with (within eps |rho| max|C| of rho.C; the
                // bias taken out again), |rho| <= rnow, and |C|^2 comes from the table the split kernel wrote.  The
                // stored terms round rho' (the factor 1.001 covers that and the table's rounding); the exact chain's
                // residual differs from it by at most (m + 1) (2^-18 + 3 * 2^-24) times the a priori bound.
                float s_code = best;
                if (bm) s_code -= __ldg(bm + code);
                const float c2 = __ldg(p.cn2 + static_cast<int64_t>(h) * MK + m * K + code);
                const float slack = 2.f * eps_m * rnow * cm + (bm ? fabsf(best) * 4.76837158203125e-7f : 0.f);
                const float ss = fmaxf(rnow * rnow - 2.f * (s_code - slack) + c2, 0.f);
                rnow = sqrtf(ss) * 1.001f + static_cast<float>(splits + 1) * 7.7e-6f * rbound;
                fence_proxy_async_smem();
                tc_fence_before();
                mbar_arrive(&bar_q[s]);
            }
        }
        if (doubt != 0 && ok) {
            // at most one entry per key: the two lists together hold every key if need be
            const unsigned int at = heavy ? p.pool_cap - 1u - atomicAdd(p.counters + 2, 1u) : atomicAdd(p.counters, 1u);
            const unsigned long long lin = static_cast<unsigned long long>(static_cast<int64_t>(u) * p.L + j);
            p.work[at] = make_uint4(static_cast<uint32_t>(lin), static_cast<uint32_t>(lin >> 32), last_rec, doubt);
        }
        if (!ok) s_err = 1;
    }
    tc_fence_before();
    __syncthreads();
    if (s_err && tid == 0) {
        if (p.status) atomicExch(p.status, VQ_WORD_TIMEOUT);
#pragma unroll 1
        for (int w = 0; w < (1 << 14); ++w) __nanosleep(256);  // let tile loads in flight land
    }
    __syncthreads();
    if (warp == C::kWarpMma) {
        __syncwarp();
        tmem_dealloc(tmem, 512u);
    }
}


// ------------------------------------------------------------------------------------------------
// Exact settlement of the doubtful keys.  A list entry is followed through the
// codebooks with the defining arithmetic - residual r_0 = k, r_{m+1} = r_m - C_m[code_m] (fp32
// subtraction) - up to its last doubtful codebook: each score is ONE fused-multiply-add chain over
// d = 0..D-1 starting from +0 (+ bias), ties go to the lowest code.  With a candidate record, one lane
// per candidate runs the chain; without one (too many candidates, no room for the record, or a code of
// an earlier codebook has changed and with it the residual) the lanes score the whole codebook.
// Bound by the latency of dependent loads: list entry -> record -> rows.  So the key, its codes and its records are fetched
// together, then all codebook rows that the residual needs and the first candidates' rows together, into shared memory.
// A whole codebook (512 KB at K = 1024, D = 128) takes one warp tens of microseconds, so four warps share it: the scan puts
// such keys on a list of their own, and a warp that changes a code leaves the key's later codebooks to its CTA.
// (us; 32 heads, D 128; before: one warp per key throughout, rows fetched as they were needed)
//   32768 bf16 keys, M4 K256: 108 -> 58;  2 x 16384, M4 K512: 300 -> 115;  5001 half keys, M1 K1024: 110 -> 43
// TEAM: warps that share an entry (1 or kAtRepairWarps); each keeps its own copy of everything but the codebook scan.
// TEAM = 1 returns the codebooks (bit m) left to the CTA.
template <int D>
struct AtRepairBuf {
    float r[D];                    // residual
    float row[kAtMaxM][D];         // C_m[code_m] as the scan left the codes
    float cand[4][D + 4];          // candidate rows (padded: four lanes read four rows)
    uint4 rec[kAtMaxM];
};

__device__ __forceinline__ void at_copy16(const float *dst, const float *src)
{
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}

template <typename KT, int D, int TEAM>
__device__ __forceinline__ uint32_t settle_key(const AtParams &p, const uint4 ent, AtRepairBuf<D> &s, float2 *team_best)
{
    constexpr unsigned kAll = 0xffffffffu;
    constexpr int PER = D / 32;    // residual elements a lane keeps up to date
    const int lane = threadIdx.x & 31, tw = TEAM > 1 ? threadIdx.x >> 5 : 0;
    const int M = p.M, K = p.K;
    const uint32_t doubt = ent.w & 0xffu, brute = (ent.w >> 8) & 0xffu;
    const int64_t lin = static_cast<int64_t>((static_cast<unsigned long long>(ent.y) << 32) | ent.x);
    const int64_t u = lin / p.L, j = lin % p.L;
    const int b = static_cast<int>(u / p.Hkv), h = static_cast<int>(u % p.Hkv);
    const KT *krow = static_cast<const KT *>(p.k) + b * p.k_sb + h * p.k_sh + j * p.k_sl;
    const float *cbh = p.cb + static_cast<int64_t>(h) * M * K * D;
    const int64_t cbase = b * p.c_sb + h * p.c_sh + j * p.c_sl;
    __syncwarp();                  // the previous entry's reads of the buffers
    const int my_code = lane < M ? load_code(p.codes, p.code_dtype, cbase + lane) : 0;
#pragma unroll
    for (int i = 0; i < PER; ++i) s.r[lane + 32 * i] = to_f32(krow[lane + 32 * i]);
    // the key's records, newest first, into a table indexed by codebook
    if (lane == 0) {
        uint32_t at = ent.z;
        for (int guard = 0; guard < kAtMaxM && at != 0xffffffffu && at < p.pool_cap; ++guard) {
            const uint4 rec = p.pool[at];
            s.rec[rec.y & 0xffu & (kAtMaxM - 1)] = rec;
            at = rec.x;
        }
    }
    if (TEAM > 1) __syncthreads();   // every warp has read the codes before one of them may rewrite them
    else __syncwarp();
    const int last = 31 - __clz(static_cast<int>(doubt | brute));   // (an entry has at least one doubtful codebook)
    auto copy_row = [&](float *dst, int m, int code) {
        if (lane < D / 4) at_copy16(dst + 4 * lane, cbh + (static_cast<int64_t>(m) * K + code) * D + 4 * lane);
    };
    auto candidate = [](const uint4 &rec, int i) { return static_cast<int>(((i < 2 ? rec.z : rec.w) >> (16 * (i & 1))) & 0xffffu); };
    auto candidates = [&](int m) { return ((doubt >> m) & 1u) ? static_cast<int>((s.rec[m].y >> 8) & 0xffu) : 0; };
    auto copy_candidates = [&](int m, int n) {
        const uint4 rec = s.rec[m];
        for (int i = 0; i < n; ++i) copy_row(s.cand[i], m, min(candidate(rec, i), K - 1));
    };
    for (int m = 0; m < last; ++m) copy_row(s.row[m], m, __shfl_sync(kAll, my_code, m));
    const int first = doubt ? __ffs(doubt) - 1 : -1;   // its candidates travel with the rows
    if (first >= 0 && candidates(first) <= 4) copy_candidates(first, candidates(first));
    bool changed = false;
    for (int m = 0; m < M && (changed || m <= last); ++m) {
        const int old = __shfl_sync(kAll, my_code, m);
        int code = old;
        const bool dm = (doubt >> m) & 1u;
        const int ncand = candidates(m);
        const bool all = changed || ((brute >> m) & 1u) || (dm && (ncand > 4 || ncand == 0));
        if (all || dm) {
            const float *cm = cbh + static_cast<int64_t>(m) * K * D;
            const float *bm = p.bias ? p.bias + (static_cast<int64_t>(h) * M + m) * K : nullptr;
            float bv = -INFINITY;
            int bi = 0x7fffffff;
            if (all) {
                bi = 0;                                     // no score above -inf (NaN scores): the first code, as in the exact kernel
                constexpr int R = 2;                        // codes per lane at a time, eight 16-byte loads of each in flight
                for (int c0 = 32 * R * tw; c0 < K; c0 += 32 * R * TEAM) {
                    float acc[R];
                    const float *row[R];
#pragma unroll
                    for (int t = 0; t < R; ++t) {
                        acc[t] = 0.f;
                        row[t] = cm + static_cast<int64_t>(min(c0 + lane + 32 * t, K - 1)) * D;
                    }
#pragma unroll 1
                    for (int d0 = 0; d0 < D; d0 += 32) {
                        float4 c4[R][8];
#pragma unroll
                        for (int t = 0; t < R; ++t)
#pragma unroll
                            for (int e = 0; e < 8; ++e) c4[t][e] = __ldg(reinterpret_cast<const float4 *>(row[t] + d0 + 4 * e));
#pragma unroll
                        for (int e = 0; e < 8; ++e) {
                            const float4 r4 = *reinterpret_cast<const float4 *>(s.r + d0 + 4 * e);
#pragma unroll
                            for (int t = 0; t < R; ++t) {
                                acc[t] = __fmaf_rn(r4.x, c4[t][e].x, acc[t]);
                                acc[t] = __fmaf_rn(r4.y, c4[t][e].y, acc[t]);
                                acc[t] = __fmaf_rn(r4.z, c4[t][e].z, acc[t]);
                                acc[t] = __fmaf_rn(r4.w, c4[t][e].w, acc[t]);
                            }
                        }
                    }
#pragma unroll
                    for (int t = 0; t < R; ++t) {
                        const int c = c0 + lane + 32 * t;
                        if (c < K) {
                            const float sc = bm ? __fadd_rn(acc[t], __ldg(bm + c)) : acc[t];
                            if (sc > bv) {      // codes come in increasing order: the first maximum stays
                                bv = sc;
                                bi = c;
                            }
                        }
                    }
                }
            } else {
                if (m != first) {
                    __syncwarp();
                    copy_candidates(m, ncand);
                }
                asm volatile("cp.async.wait_all;" ::: "memory");
                __syncwarp();
                if (lane < ncand) {
                    const int c = candidate(s.rec[m], lane);
                    if (c < K) {
                        float acc = 0.f;
#pragma unroll 8
                        for (int d = 0; d < D; d += 4) {
                            const float4 r4 = *reinterpret_cast<const float4 *>(s.r + d);
                            const float4 c4 = *reinterpret_cast<const float4 *>(s.cand[lane] + d);
                            acc = __fmaf_rn(r4.x, c4.x, acc);
                            acc = __fmaf_rn(r4.y, c4.y, acc);
                            acc = __fmaf_rn(r4.z, c4.z, acc);
                            acc = __fmaf_rn(r4.w, c4.w, acc);
                        }
                        bv = bm ? __fadd_rn(acc, __ldg(bm + c)) : acc;
                        bi = c;
                    }
                }
            }
#pragma unroll
            for (int off = 16; off >= 1; off >>= 1) {
                const float ov = __shfl_xor_sync(kAll, bv, off);
                const int oi = __shfl_xor_sync(kAll, bi, off);
                if (ov > bv || (ov == bv && oi < bi)) {
                    bv = ov;
                    bi = oi;
                }
            }
            if (TEAM > 1 && all) {   // (`all` is the same in every warp of the team: so is all that it is formed from)
                __syncthreads();
                if (lane == 0) team_best[tw] = make_float2(bv, __int_as_float(bi));
                __syncthreads();
#pragma unroll
                for (int t = 0; t < TEAM; ++t) {
                    const float2 o = team_best[t];
                    const int oi = __float_as_int(o.y);
                    if (o.x > bv || (o.x == bv && oi < bi)) {
                        bv = o.x;
                        bi = oi;
                    }
                }
            }
            if (bi != code && bi != 0x7fffffff) {
                changed = true;
                code = bi;
                if (lane == 0 && tw == 0) store_code(p.codes, p.code_dtype, cbase + m, code);
                if (TEAM == 1 && m + 1 < M) {
                    asm volatile("cp.async.wait_all;" ::: "memory");
                    return ((1u << M) - 1u) & ~((2u << m) - 1u);
                }
            }
        }
        if (m + 1 < M && (changed || m < last)) {
            asm volatile("cp.async.wait_all;" ::: "memory");
            __syncwarp();
            const bool have = code == old && m < last;       // the row that was fetched ahead
            const float *crow = cbh + (static_cast<int64_t>(m) * K + code) * D;
#pragma unroll
            for (int i = 0; i < PER; ++i) {
                const float c = have ? s.row[m][lane + 32 * i] : __ldg(crow + lane + 32 * i);
                s.r[lane + 32 * i] = __fsub_rn(s.r[lane + 32 * i], c);
            }
            __syncwarp();
        }
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    return 0u;
}

// Every key of the call, exactly, in tiles of 32 keys that share the codebook rows: for calls where so many keys tie (equal or
// collapsed codewords, residuals of zero) that scoring a codebook once per such key costs more than once per tile.  Thread (kq, cr)
// scores keys 4 kq .. 4 kq + 3 against codes cr, cr + 16, cr + 32, cr + 48 of 64 codewords, a quarter of whose columns is in shared
// memory at a time.  Bound by shared-memory loads (eight of 16 bytes per 64 FMAs).
constexpr int kBulkKeys = 32, kBulkCodes = 64;
template <typename KT, int D>
__device__ __noinline__ void settle_all(const AtParams &p, float *mem)
{
    constexpr unsigned kAll = 0xffffffffu;
    constexpr int DC = D / 4, CP = DC + 4;   // columns at a time; floats per staged row (padded: a warp's four rows lie in different banks)
    static_assert(kAtRepairWarps * 32 == kBulkKeys / 4 * 16, "thread (kq, cr)");
    float *rT = mem, *cw = rT + D * kBulkKeys;                                         // residuals [D][keys], codewords [64][DC]
    int *s_code = reinterpret_cast<int *>(cw + kBulkCodes * CP);
    float *s_v = cw;                                                                   // best scores [warp][key] and their codes, over the codewords
    int *s_i = reinterpret_cast<int *>(s_v + kAtRepairWarps * kBulkKeys);
    static_assert(sizeof(float) * (D * kBulkKeys + kBulkCodes * CP + kBulkKeys) <= kAtRepairWarps * sizeof(AtRepairBuf<D>), "shared memory");
    const int tid = threadIdx.x, warp = tid >> 5, kq = tid & 7, cr = tid >> 3;
    const int M = p.M, K = p.K;
    const int64_t per_unit = (p.L + kBulkKeys - 1) / kBulkKeys, tiles = p.pool_cap / p.L * per_unit;
    for (int64_t t = blockIdx.x; t < tiles; t += gridDim.x) {
        const int u = static_cast<int>(t / per_unit), b = u / p.Hkv, h = u % p.Hkv;
        const int64_t j0 = t % per_unit * kBulkKeys;
        const KT *kb = static_cast<const KT *>(p.k) + b * p.k_sb + h * p.k_sh;
        __syncthreads();           // the previous tile's reads
        for (int e = tid; e < kBulkKeys * D; e += kAtRepairWarps * 32) {
            const int key = e / D, d = e % D;
            rT[d * kBulkKeys + key] = j0 + key < p.L ? to_f32(kb[(j0 + key) * p.k_sl + d]) : 0.f;
        }
        for (int m = 0; m < M; ++m) {
            const float *cm = p.cb + (static_cast<int64_t>(h) * M + m) * K * D;
            const float *bm = p.bias ? p.bias + (static_cast<int64_t>(h) * M + m) * K : nullptr;
            float bv[4];
            int bi[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                bv[i] = -INFINITY;
                bi[i] = 0;         // no score above -inf (NaN scores): the first code, as in the exact kernel
            }
            for (int c0 = 0; c0 < K; c0 += kBulkCodes) {   // (K is a multiple of 128)
                float acc[4][4];   // [code][key]
#pragma unroll
                for (int i = 0; i < 16; ++i) acc[i >> 2][i & 3] = 0.f;
#pragma unroll 1
                for (int d0 = 0; d0 < D; d0 += DC) {
                    __syncthreads();   // residuals written, the previous rows read
#pragma unroll
                    for (int i = 0; i < kBulkCodes * DC / 4 / (kAtRepairWarps * 32); ++i) {
                        const int e = tid + i * kAtRepairWarps * 32, c = e / (DC / 4), q = e % (DC / 4);
                        *reinterpret_cast<float4 *>(cw + c * CP + 4 * q) = __ldg(reinterpret_cast<const float4 *>(cm + static_cast<int64_t>(c0 + c) * D + d0) + q);
                    }
                    __syncthreads();
#pragma unroll 1
                    for (int d = 0; d < DC; d += 4) {
                        float cv[4][4];
#pragma unroll
                        for (int i = 0; i < 4; ++i) {
                            const float4 c4 = *reinterpret_cast<const float4 *>(cw + (cr + 16 * i) * CP + d);
                            cv[i][0] = c4.x; cv[i][1] = c4.y; cv[i][2] = c4.z; cv[i][3] = c4.w;
                        }
#pragma unroll
                        for (int e = 0; e < 4; ++e) {
                            const float4 r4 = *reinterpret_cast<const float4 *>(rT + (d0 + d + e) * kBulkKeys + 4 * kq);
#pragma unroll
                            for (int i = 0; i < 4; ++i) {
                                acc[i][0] = __fmaf_rn(r4.x, cv[i][e], acc[i][0]);
                                acc[i][1] = __fmaf_rn(r4.y, cv[i][e], acc[i][1]);
                                acc[i][2] = __fmaf_rn(r4.z, cv[i][e], acc[i][2]);
                                acc[i][3] = __fmaf_rn(r4.w, cv[i][e], acc[i][3]);
                            }
                        }
                    }
                }
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const int c = c0 + cr + 16 * i;
#pragma unroll
                    for (int k = 0; k < 4; ++k) {
                        const float sc = bm ? __fadd_rn(acc[i][k], __ldg(bm + c)) : acc[i][k];
                        if (sc > bv[k]) {      // a thread's codes come in increasing order: the first maximum stays
                            bv[k] = sc;
                            bi[k] = c;
                        }
                    }
                }
            }
            __syncthreads();       // the last codewords have been read: the bests go over them
            auto take = [](float &v, int &i, float ov, int oi) {
                if (ov > v || (ov == v && oi < i)) {
                    v = ov;
                    i = oi;
                }
            };
#pragma unroll
            for (int i = 0; i < 4; ++i) {
#pragma unroll
                for (int off = 16; off >= 8; off >>= 1) {
                    const float ov = __shfl_xor_sync(kAll, bv[i], off);
                    const int oi = __shfl_xor_sync(kAll, bi[i], off);
                    take(bv[i], bi[i], ov, oi);
                }
                if ((tid & 31) < 8) {
                    s_v[warp * kBulkKeys + 4 * kq + i] = bv[i];
                    s_i[warp * kBulkKeys + 4 * kq + i] = bi[i];
                }
            }
            __syncthreads();
            if (tid < kBulkKeys) {
                float v = s_v[tid];
                int c = s_i[tid];
#pragma unroll
                for (int w = 1; w < kAtRepairWarps; ++w) take(v, c, s_v[w * kBulkKeys + tid], s_i[w * kBulkKeys + tid]);
                s_code[tid] = c;
                if (j0 + tid < p.L) store_code(p.codes, p.code_dtype, b * p.c_sb + h * p.c_sh + (j0 + tid) * p.c_sl + m, c);
            }
            if (m + 1 < M) {
                __syncthreads();
                const int key = tid & (kBulkKeys - 1);
                const float *crow = cm + static_cast<int64_t>(s_code[key]) * D;
                for (int q = warp; q < D / 4; q += kAtRepairWarps) {
                    const float4 x = __ldg(reinterpret_cast<const float4 *>(crow) + q);
                    float *r = rT + 4 * q * kBulkKeys + key;
                    r[0] = __fsub_rn(r[0], x.x);
                    r[kBulkKeys] = __fsub_rn(r[kBulkKeys], x.y);
                    r[2 * kBulkKeys] = __fsub_rn(r[2 * kBulkKeys], x.z);
                    r[3 * kBulkKeys] = __fsub_rn(r[3 * kBulkKeys], x.w);
                }
            }
        }
    }
}

template <typename KT, int D>
__global__ void __launch_bounds__(kAtRepairWarps * 32, 6)
assign_repair_kernel(const __grid_constant__ AtParams p)
{
    __shared__ __align__(16) AtRepairBuf<D> s_buf[kAtRepairWarps];
    __shared__ float2 s_team[kAtRepairWarps];
    __shared__ uint4 s_left[kAtLeft];          // keys whose later codebooks are left to the CTA
    __shared__ unsigned int s_nleft;
    const int warp = threadIdx.x >> 5;
    const unsigned int count = p.counters[0], heavy = p.counters[2];
    // Past this many keys with a whole codebook to score, all keys are scored in tiles (every CTA reads the same counter).  Such a
    // key takes the chip 0.07 us (K = 256) to 0.22 us (K = 1024) by itself, any key 10 ns per 1024 codes in a tile; up to two per
    // CTA they are short beside a tile's latency.  32 heads x 5001 keys, all codewords equal, M1 K1024: 40.5 -> 1.7 ms (the
    // exact kernel: 1.4 ms).  `p` is passed on by reference: as a plain parameter its copy in local memory cost every call 2 - 3 us.
    if (heavy > max(p.pool_cap / 24u, 2u * gridDim.x)) {
        settle_all<KT, D>(p, reinterpret_cast<float *>(s_buf));
        return;
    }
    if (threadIdx.x == 0) s_nleft = 0u;
    __syncthreads();
    // the long ones first: they are spread over all CTAs
    for (unsigned int e = blockIdx.x; e < heavy; e += gridDim.x) settle_key<KT, D, kAtRepairWarps>(p, p.work[p.pool_cap - 1u - e], s_buf[warp], s_team);
    for (unsigned int e = blockIdx.x * kAtRepairWarps + warp; e < count; e += gridDim.x * kAtRepairWarps) {
        uint4 ent = p.work[e];
        const uint32_t left = settle_key<KT, D, 1>(p, ent, s_buf[warp], nullptr);
        if (left == 0u) continue;
        // every code up to the changed one is settled; the codebooks after it are scored in full
        ent.z = 0xffffffffu;
        ent.w = left << 8;
        unsigned int at = 0;
        if ((threadIdx.x & 31) == 0) at = atomicAdd(&s_nleft, 1u);
        at = __shfl_sync(0xffffffffu, at, 0);
        if (at < kAtLeft) {
            if ((threadIdx.x & 31) == 0) s_left[at] = ent;
        } else {
            while (ent.w != 0u) ent.w = settle_key<KT, D, 1>(p, ent, s_buf[warp], nullptr) << 8;   // no room: one changed code at a time
        }
    }
    __syncthreads();
    const unsigned int nleft = s_nleft < kAtLeft ? s_nleft : kAtLeft;
    for (unsigned int e = 0; e < nleft; ++e) settle_key<KT, D, kAtRepairWarps>(p, s_left[e], s_buf[warp], s_team);
}

template <typename KT, int D, int NS, int CH, bool WRAP = false>
static int launch_assign_tc(const VqTensorDesc *k, const VqTensorDesc *cb, const VqTensorDesc *bias, VqTensorDesc *codes,
                            void *workspace, int32_t *status, cudaStream_t stream)
{
    using C = AtCfg<D, NS, CH>;
    const int64_t B = k->shape[0], Hkv = k->shape[1], L = k->shape[2];
    const int64_t M = cb->shape[1], K = cb->shape[2], MK = M * K;
    __nv_bfloat16 *hi = static_cast<__nv_bfloat16 *>(workspace);
    __nv_bfloat16 *lo = hi + Hkv * MK * D;
    float *cmax = reinterpret_cast<float *>(lo + Hkv * MK * D);
    float *cn2 = cmax + (Hkv * M + 63) / 64 * 64;
    unsigned int *counters = reinterpret_cast<unsigned int *>(cn2 + (Hkv * MK + 63) / 64 * 64);
    uint4 *work = reinterpret_cast<uint4 *>(counters + 64);
    uint4 *pool = work + B * Hkv * L;
    if (cudaMemsetAsync(cmax, 0, sizeof(float) * static_cast<size_t>(Hkv * M), stream) != cudaSuccess) return VQ_ELAUNCH;
    split_codebook_kernel<D><<<dim3(static_cast<unsigned>(Hkv * M), static_cast<unsigned>(K / kSplitRows)), 256, 0, stream>>>(
        static_cast<const float *>(cb->ptr), hi, lo, cmax, cn2, counters, static_cast<int>(K));
    if (launch_status() != VQ_OK) return VQ_ELAUNCH;
    CUtensorMap mk, mhi, mlo;
    const uint64_t cd[3] = {static_cast<uint64_t>(D), static_cast<uint64_t>(Hkv * MK), 1};
    const uint64_t cs[3] = {1, static_cast<uint64_t>(D), static_cast<uint64_t>(Hkv * MK * D)};
    const bool tile = k->dtype == VQ_BF16;   // the other key types are read by the scan warps
    if ((tile && !map_bhld(&mk, *k)) || !make_map(&mhi, hi, 3, cd, cs, CH) || !make_map(&mlo, lo, 3, cd, cs, CH)) return VQ_ELAUNCH;
    if (!tile) mk = mhi;
    AtParams p{};
    p.k = k->ptr;
    p.k_sb = k->stride[0]; p.k_sh = k->stride[1]; p.k_sl = k->stride[2];
    p.cb = static_cast<const float *>(cb->ptr);
    p.bias = bias ? static_cast<const float *>(bias->ptr) : nullptr;
    p.cmax = cmax;
    p.cn2 = cn2;
    p.work = work;
    p.pool = pool;
    p.counters = counters;
    p.pool_cap = static_cast<unsigned int>(B * Hkv * L < 0xfffffff0ll ? B * Hkv * L : 0xfffffff0ll);
    p.codes = codes->ptr; p.code_dtype = codes->dtype;
    p.c_sb = codes->stride[0]; p.c_sh = codes->stride[1]; p.c_sl = codes->stride[2];
    p.Hkv = static_cast<int>(Hkv); p.M = static_cast<int>(M); p.K = static_cast<int>(K);
    p.L = L;
    p.ntiles = static_cast<int>((L + kBlock - 1) / kBlock);
    p.status = status;
    p.wait_limit = wait_limit_cycles();
    static_assert(!WRAP || CH == AtCfg<D, NS, CH>::kRegion, "rounds of one chunk per use of the region");
    if (WRAP != (K / CH > C::kMaxChunks)) return VQ_EUNSUPPORTED;
    auto kern = assign_tc_kernel<KT, D, NS, CH, WRAP>;
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, C::kTotal) != cudaSuccess) return VQ_ELAUNCH;
    dim3 grid(static_cast<unsigned>((p.ntiles + NS - 1) / NS), static_cast<unsigned>(B * Hkv));
    kern<<<grid, C::kThreads, C::kTotal, stream>>>(mk, mhi, mlo, p);
    if (launch_status() != VQ_OK) return VQ_ELAUNCH;
    // the doubtful keys, exactly; the list length is only known on the device: a fixed grid walks it
    int dev = 0, sms = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return VQ_EDEVICE;
    assign_repair_kernel<KT, D><<<static_cast<unsigned>(sms * 8), kAtRepairWarps * 32, 0, stream>>>(p);
    return launch_status();
}

}  // namespace vq

extern "C" size_t vqattn_assign_workspace_bytes(int64_t B, int64_t Hkv, int64_t L, int64_t M, int64_t K, int64_t D)
{
    const size_t split = static_cast<size_t>(Hkv) * M * K * D * 2 * 2;                           // bf16 hi / lo codebooks
    const size_t norms = (static_cast<size_t>(Hkv) * M * sizeof(float) + 255) / 256 * 256;        // max row norm per codebook
    const size_t rows = (static_cast<size_t>(Hkv) * M * K * sizeof(float) + 255) / 256 * 256;    // squared norm of every row
    const size_t list = 256 + 2 * static_cast<size_t>(B) * Hkv * L * 16;   // counters; doubtful keys and candidate records, 16 bytes each, one per key at most
    return split + norms + rows + list + 256;
}

extern "C" int vqattn_assign_codes_ws(const VqTensorDesc *k, const VqTensorDesc *codebooks, const VqTensorDesc *bias,
                                      VqTensorDesc *codes, void *workspace, size_t workspace_bytes, int32_t *status_word,
                                      void *stream)
{
    using namespace vq;
    if (k == nullptr || codebooks == nullptr || codes == nullptr) return VQ_EINVAL_ARG;
    if (bias != nullptr && bias->ptr == nullptr) bias = nullptr;
    const bool shapes_ok = k->ndim == 4 && codebooks->ndim == 4;
    const int64_t D = shapes_ok ? k->shape[3] : 0, M = shapes_ok ? codebooks->shape[1] : 0, K = shapes_ok ? codebooks->shape[2] : 0;
    const int64_t align = k->dtype == VQ_BF16 ? 8 : 4;   // elements: TMA rows, 16- or 8-byte loads of the other key types
    const bool tensor_path = shapes_ok && is_act_dtype(k->dtype) && (D == 64 || D == 128) && M >= 1 && M <= kAtMaxM &&
                             K % kAtMinChunk == 0 && (K <= 512 || K == kAtMaxK) && k->stride[0] % align == 0 && k->stride[1] % align == 0 &&
                             k->stride[2] % align == 0 && k->shape[2] < (int64_t(1) << 31);
    // Few keys against few codewords: the exact kernel is one launch of a short chain, this path four (codebook split, scan,
    // repair, a memset).  Measured (us, this path / exact kernel): M*K*D = 8192: 8192 keys 25 / 11, 32768 keys 26 / 25;
    // 16384: 8192 keys 28 / 17, 32768 keys 28 / 50; 32768: 256 keys 25 / 34, 32768 keys 35 / 84.
    // M*K*D = 16384, 12288 keys, exact kernel / this path: M1 K128 25.6 / 20.5 (half 25.6 / 23.5), M2 K128 27.2 / 24; so the line runs
    // through the product as well.
    const int64_t keys = shapes_ok ? k->shape[0] * k->shape[1] * k->shape[2] : 0;
    const bool small = shapes_ok && M * K * D <= (1 << 14) && keys <= (1 << 14) && keys * (M * K * D) <= (int64_t(1) << 27);
    // half and fp32 keys without a (sufficient) workspace take the exact kernel as well
    const bool ws_ok = workspace != nullptr && reinterpret_cast<uintptr_t>(workspace) % 256 == 0 && shapes_ok &&
                       workspace_bytes >= vqattn_assign_workspace_bytes(k->shape[0], k->shape[1], k->shape[2], M, K, D);
    if (!tensor_path || (small && ws_ok) || (k->dtype != VQ_BF16 && !ws_ok)) return vqattn_assign_codes(k, codebooks, bias, codes, stream);
    // same argument checks as the exact kernel's entry point
    int st;
    if ((st = check_basic(k, 4)) != VQ_OK) return st;
    if ((st = check_basic(codebooks, 4)) != VQ_OK) return st;
    if ((st = check_basic(codes, 4)) != VQ_OK) return st;
    if (bias != nullptr && (st = check_basic(bias, 3)) != VQ_OK) return st;
    const VqTensorDesc *all[] = {k, codebooks, bias, codes};
    if ((st = check_device(all, 4)) != VQ_OK) return st;
    if (codebooks->dtype != VQ_F32 || !is_code_dtype(codes->dtype) || (bias && bias->dtype != VQ_F32)) return VQ_EINVAL_DTYPE;
    const int64_t B = k->shape[0], Hkv = k->shape[1], L = k->shape[2];
    if (codebooks->shape[0] != Hkv || codebooks->shape[3] != D) return VQ_EINVAL_SHAPE;
    if (codes->shape[0] != B || codes->shape[1] != Hkv || codes->shape[2] != L || codes->shape[3] != M) return VQ_EINVAL_SHAPE;
    if (bias && (bias->shape[0] != Hkv || bias->shape[1] != M || bias->shape[2] != K)) return VQ_EINVAL_SHAPE;
    if (!is_dense(*codebooks) || (bias && !is_dense(*bias))) return VQ_EINVAL_STRIDE;
    if (codes->dtype == VQ_U8 && K > 256) return VQ_EINVAL_DTYPE;
    if (reinterpret_cast<uintptr_t>(k->ptr) % 16 || reinterpret_cast<uintptr_t>(codebooks->ptr) % 16) return VQ_EINVAL_STRIDE;
    if (B * Hkv > 65535) return VQ_EUNSUPPORTED;
    if (!ws_ok) return VQ_EWORKSPACE;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    auto go = [&](auto key, auto dim) {
        using KT = decltype(key);
        constexpr int DD = decltype(dim)::value;
        // two key tiles per CTA share the 512 score columns of tensor memory when a codebook fits 256 of them;
        // N = 256 instructions when K is a multiple of 256
        if (K == 128) return launch_assign_tc<KT, DD, 2, 128>(k, codebooks, bias, codes, workspace, status_word, s);
        if (K == 256) return launch_assign_tc<KT, DD, 2, 256>(k, codebooks, bias, codes, workspace, status_word, s);
        // K = 512 and K = 1024: two streams, the codebook's 256-column chunks in rounds through each stream's region (the
        // candidates of a doubtful key are tracked during the scan, the earlier chunks being gone by the end)
        if (K == 512 || K == 1024) return launch_assign_tc<KT, DD, 2, 256, true>(k, codebooks, bias, codes, workspace, status_word, s);
        return launch_assign_tc<KT, DD, 1, 128>(k, codebooks, bias, codes, workspace, status_word, s);   // K = 384
    };
    using D64 = std::integral_constant<int, 64>;
    using D128 = std::integral_constant<int, 128>;
    if (k->dtype == VQ_F32) return D == 64 ? go(float(), D64()) : go(float(), D128());
    if (k->dtype == VQ_F16) return D == 64 ? go(__half(), D64()) : go(__half(), D128());
    return D == 64 ? go(__nv_bfloat16(), D64()) : go(__nv_bfloat16(), D128());
}
