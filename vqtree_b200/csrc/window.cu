// What a prefill leaves in a decode cache, in one launch: the window's rotated keys, raw keys and values copied into their
// buffers (rows behind the live ones zeroed) and the activation-dtype copy of the value sums.  Bound by memory traffic for
// long windows and by its launch for short ones; as eight separate copies, fills and a conversion it was 72 us of device time
// for 32 heads of 5001 half-precision tokens (window 1024), and eight launches: 19 us in one.
#include "vq_common.cuh"

namespace vq {

struct WindowParams {
    const uint8_t *src[3];
    uint8_t *win[3];
    int64_t s_sb[3], s_sh[3], s_sl[3];    // source strides in bytes
    int64_t n, cap, rows;                 // live rows, rows of a buffer, B * Hkv * cap
    int Hkv, vpr;                         // vectors per row
    int64_t win_items;                    // vectors of all three buffers
    const float *vsum32;
    void *vsum;
    int64_t conv_items;                   // groups of four sums
};

// V: the vector type that rows and their addresses are multiples of; I: index type (32 bits where they reach: the divisions
// were half the kernel's time)
template <typename V, typename T, typename I>
__global__ void __launch_bounds__(256) store_window_kernel(const WindowParams p)
{
    const I win_items = static_cast<I>(p.win_items), total = static_cast<I>(p.win_items + p.conv_items), rows = static_cast<I>(p.rows);
    const I cap = static_cast<I>(p.cap), vpr = static_cast<I>(p.vpr), heads = static_cast<I>(p.Hkv);
    for (I i = blockIdx.x * I(256) + threadIdx.x; i < total; i += gridDim.x * I(256)) {
        if (i >= win_items) {
            const I c = i - win_items;
            const float4 x = reinterpret_cast<const float4 *>(p.vsum32)[c];
            reinterpret_cast<uint2 *>(p.vsum)[c] = make_uint2(Pair16<T>::pack(x.x, x.y), Pair16<T>::pack(x.z, x.w));
            continue;
        }
        const I row = i / vpr, v = i - row * vpr;
        const int t = row >= 2 * rows ? 2 : row >= rows ? 1 : 0;
        const I w = row - t * rows, u = w / cap, r = w - u * cap;
        V x{};
        if (r < static_cast<I>(p.n)) {
            const I b = u / heads, h = u - b * heads;
            x = *reinterpret_cast<const V *>(p.src[t] + b * p.s_sb[t] + h * p.s_sh[t] + r * p.s_sl[t] + v * int64_t(sizeof(V)));
        }
        reinterpret_cast<V *>(p.win[t])[i - t * rows * vpr] = x;
    }
}

}  // namespace vq

extern "C" int vqattn_store_window(const VqTensorDesc *k1, const VqTensorDesc *k3, const VqTensorDesc *v, VqTensorDesc *k1_win, VqTensorDesc *k3_win,
                                   VqTensorDesc *v_win, const VqTensorDesc *vsum_f32, VqTensorDesc *vsum_act, void *stream)
{
    using namespace vq;
    const VqTensorDesc *src[3] = {k1, k3, v}, *win[3] = {k1_win, k3_win, v_win};
    if (vsum_act != nullptr && vsum_act->ptr == nullptr) vsum_act = nullptr;
    int st;
    for (int t = 0; t < 3; ++t) {
        if ((st = check_basic(src[t], 4)) != VQ_OK) return st;
        if ((st = check_basic(win[t], 4)) != VQ_OK) return st;
    }
    const VqTensorDesc *all[] = {k1, k3, v, k1_win, k3_win, v_win, vsum_act ? vsum_f32 : nullptr, vsum_act};
    if ((st = check_device(all, 8)) != VQ_OK) return st;
    const int dt = k1->dtype, esize = dt == VQ_F32 ? 4 : 2;
    if (!is_act_dtype(dt)) return VQ_EINVAL_DTYPE;
    const int64_t B = k1->shape[0], Hkv = k1->shape[1], n = k1->shape[2], D = k1->shape[3], cap = k1_win->shape[2];
    bool wide = D * esize % 16 == 0;
    WindowParams p{};
    for (int t = 0; t < 3; ++t) {
        if (src[t]->dtype != dt || win[t]->dtype != dt) return VQ_EINVAL_DTYPE;
        if (src[t]->shape[0] != B || src[t]->shape[1] != Hkv || src[t]->shape[2] != n || src[t]->shape[3] != D) return VQ_EINVAL_SHAPE;
        if (win[t]->shape[0] != B || win[t]->shape[1] != Hkv || win[t]->shape[2] != cap || win[t]->shape[3] != D || n > cap) return VQ_EINVAL_SHAPE;
        if (!is_dense(*win[t])) return VQ_EINVAL_STRIDE;
        p.src[t] = static_cast<const uint8_t *>(src[t]->ptr);
        p.win[t] = static_cast<uint8_t *>(win[t]->ptr);
        p.s_sb[t] = src[t]->stride[0] * esize; p.s_sh[t] = src[t]->stride[1] * esize; p.s_sl[t] = src[t]->stride[2] * esize;
        // (a stride over a single row is never used)
        wide = wide && reinterpret_cast<uintptr_t>(p.src[t]) % 16 == 0 && reinterpret_cast<uintptr_t>(p.win[t]) % 16 == 0 &&
               (B == 1 || p.s_sb[t] % 16 == 0) && (Hkv == 1 || p.s_sh[t] % 16 == 0) && (n == 1 || p.s_sl[t] % 16 == 0);
    }
    if (vsum_act != nullptr) {
        if ((st = check_basic(vsum_f32, 4)) != VQ_OK) return st;
        if ((st = check_basic(vsum_act, 4)) != VQ_OK) return st;
        if (vsum_f32->dtype != VQ_F32 || vsum_act->dtype != dt || dt == VQ_F32) return VQ_EINVAL_DTYPE;
        int64_t total = 1;
        for (int i = 0; i < 4; ++i) {
            if (vsum_f32->shape[i] != vsum_act->shape[i]) return VQ_EINVAL_SHAPE;
            total *= vsum_f32->shape[i];
        }
        if (!is_dense(*vsum_f32) || !is_dense(*vsum_act) || reinterpret_cast<uintptr_t>(vsum_f32->ptr) % 16 || reinterpret_cast<uintptr_t>(vsum_act->ptr) % 8)
            return VQ_EINVAL_STRIDE;
        if (total % 4) return VQ_EUNSUPPORTED;
        p.vsum32 = static_cast<const float *>(vsum_f32->ptr);
        p.vsum = vsum_act->ptr;
        p.conv_items = total / 4;
    }
    p.n = n; p.cap = cap; p.Hkv = static_cast<int>(Hkv);
    p.rows = B * Hkv * cap;
    p.vpr = static_cast<int>(wide ? D * esize / 16 : D);
    p.win_items = 3 * p.rows * p.vpr;
    int dev = 0, sms = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return VQ_EDEVICE;
    const int64_t want = (p.win_items + p.conv_items + 255) / 256, most = int64_t(sms) * 32;
    const unsigned grid = static_cast<unsigned>(want < most ? want : most);
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    const bool small = p.win_items + p.conv_items < (int64_t(1) << 31);   // (a step of the grid more still fits 32 unsigned bits)
    auto go = [&](auto vec, auto half) {
        using V = decltype(vec);
        using T = decltype(half);
        if (small) store_window_kernel<V, T, uint32_t><<<grid, 256, 0, s>>>(p);
        else store_window_kernel<V, T, int64_t><<<grid, 256, 0, s>>>(p);
    };
    if (wide) {
        if (dt == VQ_F16) go(uint4{}, __half{});
        else go(uint4{}, __nv_bfloat16{});
    } else if (dt == VQ_F16) go(uint16_t{}, __half{});
    else if (dt == VQ_BF16) go(uint16_t{}, __nv_bfloat16{});
    else go(uint32_t{}, __nv_bfloat16{});
    return launch_status();
}
