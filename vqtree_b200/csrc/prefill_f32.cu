// Fused VQ-attention prefill of fp32 inputs, register-tiled on the regular cores (single precision throughout).
//
// One CTA owns 64 query rows of one (batch, query head) and walks 64-key chunks with ONE online softmax, in this order:
//   far codebook rows     (q2 . codebook, weight cnt, value vsum)   ops/triton_fused_vq_attn.py:38-68
//   boundary keys         (q2 . k3, j < i - W)                      ops/triton_fused_local_attn_rerope.py:68-75
//   window keys           (q1 . k1, i - W <= j <= i)                ops/triton_fused_local_attn_rerope.py:45-49,76-78
// Thread (ty, tx) forms the scores of rows 4 ty .. 4 ty + 3 against keys tx, tx + 16, tx + 32, tx + 48 and owns columns
// 4 tx .. 4 tx + 3 (D = 128: and 64 + those) of the same rows' output, so maxima, denominators and P stay inside a half-warp.
// Bound by the fp32 pipe: per four elements of the head dimension 64 FMAs against eight 16-byte shared-memory loads
// (rows padded by 16 bytes: the 16 lanes of a half-warp fall into different banks).  The next chunk's keys are copied in
// (cp.async) under the softmax and the product, its values under the next scores.
// prefill_simt.cu (one warp per query row, every lane reading a different key row) stays as the cross-check kernel.
#include "vq_common.cuh"

namespace vq {

constexpr int kF32Rows = 64, kF32Keys = 64, kF32Threads = 256;

struct F32Params {
    const float *q1, *q2, *k1, *k3, *v, *codebook, *vsum, *cnt;
    float *out, *lse2;
    int64_t q_sb, q_sh, q_sl, q2_sb, q2_sh, q2_sl, o_sb, o_sh, o_sl, k_sb, k_sh, k_sl, k3_sb, k3_sh, k3_sl, v_sb, v_sh, v_sl;
    int Hq, Hkv, MK, NB, ntiles, rerope;
    int64_t L, window;
    float scale_log2;
};

template <int D>
struct F32Cfg {
    static constexpr int kPitch = D + 4;                       // floats per shared-memory row of q, k and v
    static constexpr int kPPitch = kF32Keys + 4;
    static constexpr int kQ1 = 0, kQ2 = kF32Rows * kPitch, kK = 2 * kF32Rows * kPitch, kV = kK + kF32Keys * kPitch,
                         kP = kV + kF32Keys * kPitch, kW = kP + kF32Rows * kPPitch, kFloats = kW + kF32Keys;
    static constexpr int kBytes = kFloats * 4;
};

// 64 rows of D floats into shared memory; rows from `valid` on are filled with zeros and not read
template <int D>
__device__ __forceinline__ void f32_copy_rows(float *dst, const float *src, int64_t stride, int64_t valid)
{
    constexpr int LPR = D / 4;                                 // 16-byte pieces of a row
#pragma unroll
    for (int i = 0; i < kF32Rows * LPR / kF32Threads; ++i) {
        const int e = i * kF32Threads + threadIdx.x, r = e / LPR, c = e % LPR;
        const uint32_t d = static_cast<uint32_t>(__cvta_generic_to_shared(dst + r * F32Cfg<D>::kPitch + 4 * c));
        const bool on = r < valid;
        const float *s = src + (on ? r : 0) * stride + 4 * c;
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(s), "r"(on ? 16 : 0) : "memory");
    }
}
__device__ __forceinline__ void f32_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void f32_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

template <int D>
__global__ void __launch_bounds__(kF32Threads, D == 64 ? 2 : 1) prefill_f32_kernel(F32Params p)
{
    using C = F32Cfg<D>;
    constexpr int NC = D / 64;                                 // column groups of four per thread
    extern __shared__ __align__(16) float f32_smem[];
    float *sm = f32_smem;
    const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
    const int t = p.ntiles - 1 - static_cast<int>(blockIdx.x);    // heavy tiles first
    const int bh = blockIdx.y, b = bh / p.Hq, hq = bh % p.Hq, hk = hq / (p.Hq / p.Hkv);
    const int64_t u = static_cast<int64_t>(b) * p.Hkv + hk;
    const int64_t i0 = static_cast<int64_t>(t) * kF32Rows;
    const int wt = static_cast<int>(p.window / kF32Keys);      // window in chunks
    const int kb0 = t / 2 - wt / 2;                            // boundary block of 128 keys (exists when >= 0)
    const int cw = t - wt;                                     // chunk in which the window of these rows begins
    const int n_far = kb0 >= 1 && p.MK > 0 ? p.MK / kF32Keys : 0;
    // chunks before the window, scored with (q2, k3): those in front of cw, and with ReRoPE cw itself (masked)
    const int n_a = kb0 >= 0 ? cw - 2 * kb0 + (p.rerope ? 1 : 0) : 0;
    const int first_b = cw > 0 ? cw : 0;
    const int n = n_far + n_a + (t - first_b + 1);

    const float *q1 = p.q1 + b * p.q_sb + hq * p.q_sh + i0 * p.q_sl, *q2 = p.q2 + b * p.q2_sb + hq * p.q2_sh + i0 * p.q2_sl;
    const float *k1 = p.k1 + b * p.k_sb + hk * p.k_sh, *k3 = p.k3 + b * p.k3_sb + hk * p.k3_sh, *v = p.v + b * p.v_sb + hk * p.v_sh;
    const float *cbk = p.codebook + static_cast<int64_t>(hk) * p.MK * D;
    const int64_t far_row = (u * p.NB + kb0 - 1) * p.MK;       // first row of the snapshot (read only when n_far > 0)
    // chunk c of the list: 0 .. n_far - 1 far, then the (q2, k3) chunks, then the (q1, k1) chunks
    auto key_chunk = [&](int c) { return c < n_far + n_a ? 2 * kb0 + (c - n_far) : first_b + (c - n_far - n_a); };
    auto copy_keys = [&](int c) {
        if (c < n_far) {
            f32_copy_rows<D>(sm + C::kK, cbk + static_cast<int64_t>(c) * kF32Keys * D, D, kF32Keys);
            if (tid < kF32Keys / 4)
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(static_cast<uint32_t>(__cvta_generic_to_shared(sm + C::kW + 4 * tid))),
                             "l"(p.cnt + far_row + c * kF32Keys + 4 * tid) : "memory");
        } else {
            const int64_t j0 = static_cast<int64_t>(key_chunk(c)) * kF32Keys;
            if (c < n_far + n_a) f32_copy_rows<D>(sm + C::kK, k3 + j0 * p.k3_sl, p.k3_sl, p.L - j0);
            else f32_copy_rows<D>(sm + C::kK, k1 + j0 * p.k_sl, p.k_sl, p.L - j0);
        }
        f32_commit();
    };
    auto copy_values = [&](int c) {
        if (c < n_far) {
            f32_copy_rows<D>(sm + C::kV, p.vsum + (far_row + static_cast<int64_t>(c) * kF32Keys) * D, D, kF32Keys);
        } else {
            const int64_t j0 = static_cast<int64_t>(key_chunk(c)) * kF32Keys;
            f32_copy_rows<D>(sm + C::kV, v + j0 * p.v_sl, p.v_sl, p.L - j0);
        }
        f32_commit();
    };
    f32_copy_rows<D>(sm + C::kQ1, q1, p.q_sl, p.L - i0);
    if (p.rerope) f32_copy_rows<D>(sm + C::kQ2, q2, p.q2_sl, p.L - i0);
    copy_keys(0);
    copy_values(0);

    float m[4], l[4], acc[4][4 * NC];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        m[i] = -INFINITY;
        l[i] = 0.f;
#pragma unroll
        for (int c = 0; c < 4 * NC; ++c) acc[i][c] = 0.f;
    }
#pragma unroll 1
    for (int c = 0; c < n; ++c) {
        const bool far = c < n_far, use2 = c < n_far + n_a;
        f32_wait<1>();                                         // this chunk's keys (its values may still be on their way)
        __syncthreads();
        // ---- scores
        float s[4][4];
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) s[i][j] = 0.f;
        {
            const float *qs = sm + (use2 && p.rerope ? C::kQ2 : C::kQ1) + 4 * ty * C::kPitch, *ks = sm + C::kK + tx * C::kPitch;
#pragma unroll 4
            for (int d = 0; d < D; d += 4) {
                float4 qv[4], kv[4];
#pragma unroll
                for (int i = 0; i < 4; ++i) qv[i] = *reinterpret_cast<const float4 *>(qs + i * C::kPitch + d);
#pragma unroll
                for (int j = 0; j < 4; ++j) kv[j] = *reinterpret_cast<const float4 *>(ks + 16 * j * C::kPitch + d);
#pragma unroll
                for (int i = 0; i < 4; ++i)
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        s[i][j] = fmaf(qv[i].x, kv[j].x, s[i][j]);
                        s[i][j] = fmaf(qv[i].y, kv[j].y, s[i][j]);
                        s[i][j] = fmaf(qv[i].z, kv[j].z, s[i][j]);
                        s[i][j] = fmaf(qv[i].w, kv[j].w, s[i][j]);
                    }
            }
        }
        float w[4] = {1.f, 1.f, 1.f, 1.f};
        if (far) {
#pragma unroll
            for (int j = 0; j < 4; ++j) w[j] = sm[C::kW + tx + 16 * j];
        }
        __syncthreads();                                       // keys and counts have been read
        if (c + 1 < n) copy_keys(c + 1);
        else f32_commit();
        // ---- masks: codes without members; keys on the wrong side of the window's edge; future keys
        const int kc = far ? 0 : key_chunk(c);
        const bool edge_a = use2 && !far && kc == cw, edge_b = !use2 && kc == cw && p.rerope, diag = !use2 && kc == t;
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const int row = 4 * ty + i, col = tx + 16 * j;
                const bool on = far ? w[j] > 0.f : !((edge_a && col >= row) || (edge_b && col < row) || (diag && col > row));
                s[i][j] = on ? s[i][j] * p.scale_log2 : -INFINITY;
            }
        // ---- online softmax of the four rows (16 lanes share a row)
        float *ps = sm + C::kP + 4 * ty * C::kPPitch;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            float mx = fmaxf(fmaxf(s[i][0], s[i][1]), fmaxf(s[i][2], s[i][3]));
#pragma unroll
            for (int off = 8; off >= 1; off >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, off));
            const float m_new = fmaxf(m[i], mx), m_safe = m_new == -INFINITY ? 0.f : m_new;   // (-inf: no key so far)
            const float alpha = exp2f(m[i] - m_safe);          // m = -inf -> 0
            float sum = 0.f;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const float pv = exp2f(s[i][j] - m_safe);      // excluded: 0
                sum = fmaf(pv, w[j], sum);
                ps[i * C::kPPitch + tx + 16 * j] = pv;
            }
#pragma unroll
            for (int off = 8; off >= 1; off >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, off);
            l[i] = fmaf(l[i], alpha, sum);
            m[i] = m_new;
#pragma unroll
            for (int cc = 0; cc < 4 * NC; ++cc) acc[i][cc] *= alpha;
        }
        f32_wait<1>();                                         // this chunk's values (the next keys may still be on their way)
        __syncthreads();
        // ---- output += P V; a weight of zero leaves the sum alone whatever the value (infinities in excluded rows)
#pragma unroll 2
        for (int k0 = 0; k0 < kF32Keys; k0 += 4) {
            float4 pr[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) pr[i] = *reinterpret_cast<const float4 *>(ps + i * C::kPPitch + k0);
#pragma unroll
            for (int kk = 0; kk < 4; ++kk) {
                float vv[4 * NC];
#pragma unroll
                for (int g = 0; g < NC; ++g) {
                    const float4 x = *reinterpret_cast<const float4 *>(sm + C::kV + (k0 + kk) * C::kPitch + 64 * g + 4 * tx);
                    vv[4 * g] = x.x; vv[4 * g + 1] = x.y; vv[4 * g + 2] = x.z; vv[4 * g + 3] = x.w;
                }
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const float pv = kk == 0 ? pr[i].x : kk == 1 ? pr[i].y : kk == 2 ? pr[i].z : pr[i].w;
                    if (pv != 0.f) {
#pragma unroll
                        for (int cc = 0; cc < 4 * NC; ++cc) acc[i][cc] = fmaf(pv, vv[cc], acc[i][cc]);
                    }
                }
            }
        }
        __syncthreads();                                       // values and P have been read
        if (c + 1 < n) copy_values(c + 1);
        else f32_commit();
    }
    f32_wait<0>();
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int64_t row = i0 + 4 * ty + i;
        if (row >= p.L) continue;
        const float inv = 1.f / l[i];
        float *o = p.out + b * p.o_sb + hq * p.o_sh + row * p.o_sl + 4 * tx;
#pragma unroll
        for (int g = 0; g < NC; ++g)
            *reinterpret_cast<float4 *>(o + 64 * g) = make_float4(acc[i][4 * g] * inv, acc[i][4 * g + 1] * inv, acc[i][4 * g + 2] * inv, acc[i][4 * g + 3] * inv);
        if (p.lse2 && tx == 0) p.lse2[static_cast<int64_t>(bh) * p.L + row] = m[i] + log2f(l[i]);
    }
}

template <int D>
static int launch_f32(const F32Params &p, int64_t B, cudaStream_t stream)
{
    auto kern = prefill_f32_kernel<D>;
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, F32Cfg<D>::kBytes) != cudaSuccess) return VQ_ELAUNCH;
    kern<<<dim3(static_cast<unsigned>(p.ntiles), static_cast<unsigned>(B * p.Hq)), kF32Threads, F32Cfg<D>::kBytes, stream>>>(p);
    return launch_status();
}

int launch_prefill_f32(const VqPrefillArgs *a, cudaStream_t stream)
{
    F32Params p{};
    auto f = [](const VqTensorDesc &t) { return static_cast<const float *>(t.ptr); };
    p.q1 = f(a->q1); p.q2 = f(a->q2); p.k1 = f(a->k1); p.k3 = f(a->k3); p.v = f(a->v);
    p.codebook = f(a->codebook); p.vsum = f(a->vsum); p.cnt = f(a->cnt);
    p.out = static_cast<float *>(a->out.ptr); p.lse2 = static_cast<float *>(a->lse2.ptr);
    p.q_sb = a->q1.stride[0]; p.q_sh = a->q1.stride[1]; p.q_sl = a->q1.stride[2];
    p.q2_sb = a->q2.stride[0]; p.q2_sh = a->q2.stride[1]; p.q2_sl = a->q2.stride[2];
    p.o_sb = a->out.stride[0]; p.o_sh = a->out.stride[1]; p.o_sl = a->out.stride[2];
    p.k_sb = a->k1.stride[0]; p.k_sh = a->k1.stride[1]; p.k_sl = a->k1.stride[2];
    p.k3_sb = a->k3.stride[0]; p.k3_sh = a->k3.stride[1]; p.k3_sl = a->k3.stride[2];
    p.v_sb = a->v.stride[0]; p.v_sh = a->v.stride[1]; p.v_sl = a->v.stride[2];
    p.Hq = static_cast<int>(a->q1.shape[1]); p.Hkv = static_cast<int>(a->k1.shape[1]);
    p.L = a->q1.shape[2];
    p.MK = a->codebook.ptr ? static_cast<int>(a->codebook.shape[1]) : 0;
    p.NB = a->cnt.ptr ? static_cast<int>(a->cnt.shape[2]) : 0;
    p.ntiles = static_cast<int>((p.L + kF32Rows - 1) / kF32Rows);
    p.window = a->window;
    auto same = [](const VqTensorDesc &x, const VqTensorDesc &y) {
        return x.ptr == y.ptr && x.stride[0] == y.stride[0] && x.stride[1] == y.stride[1] && x.stride[2] == y.stride[2];
    };
    p.rerope = same(a->q1, a->q2) && same(a->k1, a->k3) ? 0 : 1;
    const int D = static_cast<int>(a->q1.shape[3]);
    const float scale = a->scale > 0.f ? a->scale : 1.0f / sqrtf(static_cast<float>(D));
    p.scale_log2 = scale * 1.4426950408889634f;
    return D == 64 ? launch_f32<64>(p, a->q1.shape[0], stream) : launch_f32<128>(p, a->q1.shape[0], stream);
}

}  // namespace vq
