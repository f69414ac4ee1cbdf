"""GPU tests of the branches that a call's type, size or alignment selects, at the sizes where each can go wrong."""
import pytest
import torch

from vqtree_b200.native import VqError

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def api():
    from vqtree_b200 import api as _api
    return _api


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _rn(g, *s):
    return torch.randn(*s, generator=g, device="cuda")


# half and fp32 keys on the tensor cores (two bf16 terms from the start): the same codes as the exact kernel, whole numbers; (127, 64, 2,
# 128) is small enough to be handed to that kernel
@pytest.mark.parametrize("dtype", [torch.float16, torch.float32])
@pytest.mark.parametrize("L,D,M,K", [(1, 64, 3, 128), (127, 64, 2, 128), (127, 64, 3, 128), (515, 64, 3, 128), (1, 128, 2, 128), (640, 64, 2, 512), (513, 64, 2, 1024), (385, 128, 2, 128), (129, 128, 4, 256), (257, 128, 8, 256), (700, 64, 3, 384),
                                     (640, 128, 2, 512), (1025, 128, 1, 1024)])
def test_assign_half_and_fp32_keys_equal_the_exact_kernel(api, dtype, L, D, M, K):
    g = _gen(L + K)
    cb = _rn(g, 3, M, K, D) * D ** -0.25
    cb[:, :, 1::8] = cb[:, :, 0::8] * (1 + 2.0 ** -18)        # near-twins: inside the bound of the approximate scores
    for scale in (1.0, 300.0):
        k = (_rn(g, 2, L, 3, D) * scale).to(dtype)
        k[:, L // 2] = 0                                       # every score ties
        k = k.transpose(1, 2)
        got = api.assign_codes(k, cb, out_dtype=torch.int32)
        want = api.assign_codes(k, cb, out_dtype=torch.int32, impl="simt")
        api.check_status()
        assert torch.equal(got, want), f"{int((got != want).sum())} codes differ"


# keys without a finite error bound (infinities, NaN, squares that overflow) or with a vanishing one (squares that underflow)
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
@pytest.mark.parametrize("M,K", [(2, 256), (1, 1024)])
def test_assign_extreme_keys_equal_the_exact_kernel(api, dtype, M, K):
    g = _gen(K)
    cb = _rn(g, 2, M, K, 128) * 128 ** -0.25
    cb[:, :, 1::8] = cb[:, :, 0::8] * (1 + 2.0 ** -18)
    k = _rn(g, 2, 2, 400, 128)
    big, tiny = (3e4, 1e-7) if dtype == torch.float16 else (1e30, 1e-24)
    k[:, :, 0:8, 3] = float("inf")
    k[:, :, 8:16, 5] = -float("inf")
    k[:, :, 16:24, 7] = float("nan")
    k[:, :, 24:32] = float("nan")
    k[:, :, 32:128] *= big
    k[:, :, 128:256] *= tiny
    k = k.to(dtype)
    got = api.assign_codes(k, cb, out_dtype=torch.int32)
    want = api.assign_codes(k, cb, out_dtype=torch.int32, impl="simt")
    api.check_status()
    assert torch.equal(got, want), f"{int((got != want).sum())} codes differ"


# keys that tie with many codes: zero keys (padding; their code is 0 without a second look) among others, with the first codeword finite
# or not and with a bias; collapsed codebooks, where more keys have a whole codebook to score than is done one by one
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
@pytest.mark.parametrize("D,M,K", [(64, 3, 128), (128, 2, 256), (128, 1, 1024), (64, 2, 512)])
def test_assign_tied_keys_equal_the_exact_kernel(api, dtype, D, M, K):
    g = _gen(D + K)
    L = 1381
    cb = _rn(g, 2, M, K, D) * D ** -0.25
    k = _rn(g, 2, L, 2, D).to(dtype).transpose(1, 2)
    k[:, :, L // 3: L // 2] = 0
    k[:, :, L // 2, D - 1] = -0.0
    k[:, 1, 7] = 0
    k[:, 1, 7, 5] = 6e-8 if dtype == torch.float16 else 1e-30      # not zero, though its square is
    bad = cb.clone()
    bad[:, 0, 0, 3] = float("nan")
    bad[1, 0, 1, 3] = float("inf")
    flat = cb.clone()
    flat[:, :, :] = flat[:, :, :1]
    flat[:, :, K // 2:, 0] += 2.0 ** -20
    bias = _rn(g, 2, M, K)
    for books, b in ((cb, None), (bad, None), (flat, None), (torch.zeros_like(cb), None), (cb, bias), (flat, bias * 0)):
        got = api.assign_codes(k, books, b, out_dtype=torch.int32)
        want = api.assign_codes(k, books, b, out_dtype=torch.int32, impl="simt")
        api.check_status()
        assert torch.equal(got, want), f"{int((got != want).sum())} codes differ"


# more keys whose code the repair changes than a CTA can leave to its four warps (64 each): twins 2^-20 apart, of which the scan, whose
# scores they share, takes the lower and the defining arithmetic the larger
def test_assign_changes_more_codes_than_are_left_to_a_cta(api):
    g = _gen(11)
    cb = _rn(g, 8, 3, 128, 64) * 64 ** -0.25
    cb[:, :, 1::2] = cb[:, :, 0::2] * (1 + 2.0 ** -20)
    k = _rn(g, 1, 8, 24000, 64).bfloat16()
    got = api.assign_codes(k, cb, out_dtype=torch.int32)
    want = api.assign_codes(k, cb, out_dtype=torch.int32, impl="simt")
    api.check_status()
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    assert int((want[..., 0] % 2).sum()) > 64 * 8 * sms
    assert torch.equal(got, want), f"{int((got != want).sum())} codes differ"


# sorted aggregates of half and fp32 values: the same sums bit for bit as the kernel without a workspace
@pytest.mark.parametrize("dtype", [torch.float16, torch.float32])
@pytest.mark.parametrize("L,D,M,K", [(128, 64, 1, 128), (390, 128, 2, 256), (1024, 64, 3, 64), (640, 128, 1, 1024)])
def test_sorted_aggregates_of_half_and_fp32_values(api, dtype, L, D, M, K):
    g = _gen(L * 3 + K)
    v = _rn(g, 2, L, 2, D).to(dtype).transpose(1, 2)
    codes = torch.randint(0, K, (2, 2, L, M), generator=g, device="cuda", dtype=torch.int32)
    codes[:, 1, : L // 2] = 5                                   # more keys of one code than a warp stages at once
    nb = L // 128
    want = api.build_aggregates(codes, v, K, nb, impl="scan")
    got = api.build_aggregates(codes, v, K, nb, state_blocks=nb)
    plain = api.build_aggregates(codes, v, K, nb)                # few blocks: the kernel without a workspace
    api.check_status()
    for a, p, b in zip(got[:2], plain, want):
        assert torch.equal(a, b) and torch.equal(p, b)
    wrong = codes.clone()
    wrong[1, 1, 100, 0] = K                                     # left out, and reported on either path
    bad = api.build_aggregates(wrong, v, K, nb)
    with pytest.raises(VqError):
        api.check_status()
    assert float(bad[0][:, :, -1].sum()) == float(plain[0][:, :, -1].sum()) - 1
    cnt, vs = torch.zeros_like(got[2]), torch.zeros_like(got[3])
    api.cache_advance(codes[:, :, : nb * 128], v[:, :, : nb * 128], K, cnt, vs)
    assert torch.equal(got[2], cnt) and torch.equal(got[3], vs)


# rows gathered as 16-byte vectors (64, 128, 256, 512 bytes a row; the first falls back to single elements), indexes outside the array;
# 2358 rows, which go element by element, and 4662
@pytest.mark.parametrize("C", [131, 259])
@pytest.mark.parametrize("dtype,D", [(torch.bfloat16, 32), (torch.bfloat16, 64), (torch.float16, 128), (torch.float32, 128)])
@pytest.mark.parametrize("idx", [torch.int64, torch.int32])
def test_gather_aggregates_moves_whole_rows(api, dtype, D, idx, C):
    g = _gen(D)
    B, H, L, NB = 2, 3, 300, 3
    v = _rn(g, B, H, L + 1, D).to(dtype)
    vi = torch.randint(-2, L + 4, (B, H, NB + 1, C), generator=g, device="cuda").to(idx)
    cnt = torch.randint(0, 3, (B, H, NB, C), generator=g, device="cuda").float()
    for c in (None, cnt):
        got = api.gather_aggregates(v, vi, NB, c)
        at = vi[:, :, :NB].long()
        ok = (at >= 0) & (at <= L) & (torch.ones_like(cnt, dtype=torch.bool) if c is None else c > 0)
        want = torch.gather(v, 2, at.clamp(0, L).reshape(B, H, -1, 1).expand(-1, -1, -1, D)).reshape(B, H, NB, C, D)
        assert torch.equal(got, torch.where(ok[..., None], want, torch.zeros_like(want)))


# the fp32 kernel (64-row tiles, 64-key chunks) against the one-warp-per-row kernel: edges of tiles, chunks, the window and the
# boundary block; codes without members whose codeword scores highest; infinities behind weights of zero.  Both are fp32 chains:
# scores of at most 16 (log2 units) carry D + 2 roundings of 2^-24 at most, sums of n <= 2000 weights as many: 2e-5 is above both.
@pytest.mark.parametrize("L,W,D,Hq,Hkv,M,K", [(1, 128, 64, 1, 1, 1, 128), (63, 128, 128, 2, 1, 1, 128), (129, 128, 64, 2, 2, 1, 128), (257, 128, 128, 4, 2, 2, 128),
                                              (320, 128, 64, 3, 1, 1, 128), (449, 256, 64, 2, 1, 2, 256), (833, 128, 128, 2, 2, 1, 384), (1024, 512, 64, 4, 4, 2, 256)])
@pytest.mark.parametrize("rerope", [False, True])
def test_prefill_fp32_equals_the_row_kernel(api, L, W, D, Hq, Hkv, M, K, rerope):
    g = _gen(L + D)
    q1, q2 = (_rn(g, 2, L, Hq, D).transpose(1, 2) for _ in range(2))
    k1, k3, v = (_rn(g, 2, Hkv, L, D) for _ in range(3))
    if not rerope:
        q2, k3 = q1, k1
    v[:, :, L - 1, 0] = float("inf")                        # the last key: weight zero in every other row
    nb = api.far_blocks(L, W)
    act = cnt = vs = None
    if nb:
        act = _rn(g, Hkv, M * K, D) * D ** -0.25
        act[:, 3] *= 30
        cnt = torch.randint(0, 4, (2, Hkv, nb, M * K), generator=g, device="cuda").float()
        cnt[..., 3] = 0
        vs = _rn(g, 2, Hkv, nb, M * K, D) * cnt[..., None]
        vs[..., 3, :] = float("inf")
    got, lse = api.prefill_from_aggregates(q1, q2, k1, k3, v, act, cnt, vs, W, return_lse=True)
    want, lse_w = api.prefill_from_aggregates(q1, q2, k1, k3, v, act, cnt, vs, W, return_lse=True, impl="simt")
    assert torch.equal(torch.isinf(got), torch.isinf(want))
    ok = ~torch.isinf(want)
    assert (got[ok] - want[ok]).abs().max() < 2e-5 and (lse - lse_w).abs().max() < 2e-5


# the window a prefill leaves behind: whole vectors, and single elements where rows or addresses are no multiples of 16 bytes
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
@pytest.mark.parametrize("n,cap,D,pad", [(1, 3, 64, 0), (130, 512, 128, 0), (57, 57, 128, 3), (9, 20, 40, 1)])
def test_store_window_copies_and_zeroes(api, dtype, n, cap, D, pad):
    g = _gen(n)
    src = [_rn(g, 2, n + 5, 3, D + pad).to(dtype).transpose(1, 2)[:, :, 5:, pad:] for _ in range(3)]
    win = [torch.full((2, 3, cap, D), 7.0, dtype=dtype, device="cuda") for _ in range(3)]
    vs = _rn(g, 2, 3, 8, D) * 1e5
    act = None if dtype == torch.float32 else torch.empty(vs.shape, dtype=dtype, device="cuda")
    api.store_window(*src, *win, vs if act is not None else None, act)
    for s, w in zip(src, win):
        assert torch.equal(w[:, :, :n], s) and not w[:, :, n:].any()
    assert act is None or torch.equal(act, vs.to(dtype))


# indices past 32 bits: 3 x 2^31 / 3 single elements and more (5 GB in all)
def test_store_window_past_32_bit_indices(api):
    D, n = 41, 1 << 20
    cap = (1 << 31) // (3 * D) + 1000
    src = _rn(_gen(1), 1, 1, n, D).half()
    win = [torch.full((1, 1, cap, D), 7.0, dtype=torch.half, device="cuda") for _ in range(3)]
    api.store_window(src, src, src, *win)
    for w in win:
        assert torch.equal(w[:, :, :n], src) and int(w[:, :, n:].count_nonzero()) == 0


# what a prefill leaves in the cache when its tensors carry tangents, are negated lazily, or have no rows
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_update_prefill_of_tensors_that_a_kernel_cannot_read(dtype):
    from torch.autograd import forward_ad as fw

    from vqtree_b200.attn_vq import VectorQuantizedReRoPECache
    g = _gen(3)
    k, raw, v, tan = (_rn(g, 2, 2, 100, 64).to(dtype) for _ in range(4))
    cnt, vs = _rn(g, 2, 2, 128), _rn(g, 2, 2, 128, 64)

    def cache():
        return VectorQuantizedReRoPECache(128, torch.zeros(2, 1, 128, 64, device="cuda"))

    c = cache()
    with fw.dual_level():
        c.update_prefill(cnt, vs, fw.make_dual(k, tan), v, 0, 100, {"key_unrotated": raw})
        got = fw.unpack_dual(c.key_buffers[0])
        assert torch.equal(got.primal, k) and torch.equal(got.tangent, tan)
    c = cache()
    c.update_prefill(cnt, vs, torch._neg_view(k), v, 0, 100, {"key_unrotated": raw})
    assert torch.equal(c.key_buffers[0], -k)
    c = cache()
    c.update_prefill(cnt[:0], vs[:0], k[:0], v[:0], 0, 100, {"key_unrotated": raw[:0]})
    assert c.key_buffers[0].shape == (0, 2, 100, 64)


# decode tiles start at row 0 for the rows before n_bd and at row n_bd for the others: edges of tiles on either side, nothing on
# one side, nothing but far rows.  Reference: the same weights in fp32; P and the output are rounded to bf16 (2^-9 each of values
# of order one), hence the 2e-2 of the bf16 bars.
@pytest.mark.parametrize("n,n_bd,far", [(1, 0, False), (1, 1, True), (128, 127, True), (129, 128, False), (257, 1, True), (300, 129, True), (256, 256, True), (0, 0, True)])
@pytest.mark.parametrize("G", [1, 4])
def test_decode_rows_on_either_side_of_the_boundary(api, n, n_bd, far, G):
    g = _gen(n * 7 + n_bd)
    B, H, D, MK = 2, 3, 128, 256
    q1, q2 = (_rn(g, B, H * G, D).bfloat16() for _ in range(2))
    k1, k3, v = (_rn(g, B, H, n + 5, D).bfloat16() for _ in range(3))
    act = _rn(g, H, MK, D).bfloat16() if far else None
    cnt = torch.randint(0, 3, (B, H, MK), generator=g, device="cuda").float() if far else None
    vs = (_rn(g, B, H, MK, D) * cnt[..., None]).bfloat16() if far else None
    got = api.vq_attention_decode(q1, q2, k1, k3, v, act, cnt, vs, n_valid=n, n_bd=n_bd).float()
    api.check_status()
    q1f, q2f = (t.float().view(B, H, G, D) for t in (q1, q2))
    s = [torch.einsum("bhgd,bhnd->bhgn", q2f, k3[:, :, :n_bd].float()), torch.einsum("bhgd,bhnd->bhgn", q1f, k1[:, :, n_bd:n].float())]
    w, val = [torch.ones(B, H, n, device="cuda")], [v[:, :, :n].float()]
    if far:
        s.append(torch.einsum("bhgd,hnd->bhgn", q2f, act.float()).masked_fill((cnt == 0)[:, :, None], float("-inf")))
        w.append(cnt)
        val.append(vs.float())
    p = torch.exp(torch.cat(s, -1) * D ** -0.5 - torch.cat(s, -1).amax(-1, keepdim=True) * D ** -0.5)
    want = torch.einsum("bhgn,bhnd->bhgd", p, torch.cat(val, 2)) / (p * torch.cat(w, 2)[:, :, None]).sum(-1, keepdim=True)
    assert (got.view(B, H, G, D) - want).abs().max() < 2e-2 * max(1.0, float(want.abs().max()))


# one head of a position per thread, or four (the last shape): head counts with a remainder, both memory orders, explicit positions; same bits as one tensor
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
@pytest.mark.parametrize("Hq,Hkv,L,D", [(1, 1, 1, 64), (5, 3, 77, 128), (8, 4, 130, 64), (13, 6, 590, 128)])
@pytest.mark.parametrize("heads_inner", [False, True])
def test_rope_qk_equals_rope(api, dtype, Hq, Hkv, L, D, heads_inner):
    g = _gen(Hq + L)
    q, k = ((_rn(g, 2, L, H, D).transpose(1, 2) if heads_inner else _rn(g, 2, H, L, D)).to(dtype) for H in (Hq, Hkv))
    pos = torch.randint(0, 500, (2, L), generator=g, device="cuda")
    for positions in (None, pos):
        q1, q2, k1 = api.rope_qk(q, k, positions, const_pos=300, n_pos=600, like_input=heads_inner)
        w1, w2 = api.rope(q, positions, const_pos=300, n_pos=600)
        assert torch.equal(q1, w1) and torch.equal(q2, w2) and torch.equal(k1, api.rope(k, positions, n_pos=600)[0])
    api.check_status()


# the two forms of the 16-bit prefill (128-key steps; 64-key steps for short tiles on grids that fill the chip) on either side of
# each line between them, ragged lengths, empty codes, grouped heads; keys that grow along the sequence, so that references are raised in
# many items and in either half of one.  Reference: the fp32 row kernel; P and the output are rounded to 8 (11) bits, hence the bars.
@pytest.mark.parametrize("growing", [False, True])
@pytest.mark.parametrize("dtype,bar", [(torch.bfloat16, 2e-2), (torch.float16, 2.5e-3)])
@pytest.mark.parametrize("B,Hq,Hkv,L,W,MK,D", [(1, 1, 1, 100, 128, 128, 64), (2, 2, 1, 129, 128, 128, 128), (1, 4, 2, 700, 128, 256, 128), (1, 3, 3, 1025, 256, 640, 64),
                                               (3, 32, 8, 300, 128, 128, 128), (2, 16, 4, 1200, 128, 1536, 128), (2, 16, 4, 1200, 128, 1536, 64), (2, 24, 4, 577, 256, 256, 64)])
@pytest.mark.parametrize("rerope", [False, True])
def test_prefill_forms_agree_with_the_row_kernel(api, dtype, bar, B, Hq, Hkv, L, W, MK, D, rerope, growing):
    g = _gen(L + MK)
    q1, q2 = (_rn(g, B, Hq, L, D).to(dtype) for _ in range(2))
    k1, k3, v = (_rn(g, B, Hkv, L, D).to(dtype) for _ in range(3))
    if growing:
        ramp = torch.linspace(0.05, 4.0, L, device="cuda")[:, None]
        k1, k3 = (k1 * ramp).to(dtype), (k3 * ramp).to(dtype)
    if not rerope:
        q2, k3 = q1, k1
    nb = api.far_blocks(L, W)
    act = cnt = vs = None
    if nb:
        act = (_rn(g, Hkv, MK, D) * D ** -0.25).to(dtype)
        cnt = torch.randint(0, 4, (B, Hkv, nb, MK), generator=g, device="cuda").float()
        vs = (_rn(g, B, Hkv, nb, MK, D) * cnt[..., None]).to(dtype)
    got, lse = api.prefill_from_aggregates(q1, q2, k1, k3, v, act, cnt, vs, W, return_lse=True)
    want, lse_w = api.prefill_from_aggregates(q1, q2, k1, k3, v, act, cnt, vs, W, return_lse=True, impl="simt")
    api.check_status()
    assert (got.float() - want.float()).abs().max() <= bar * max(1.0, float(want.float().abs().max())) and (lse - lse_w).abs().max() < 1e-4 * max(1.0, float(lse_w.abs().max()) / 10)


# a row whose largest score lies in the second half of its first 128 keys, up to 2^8 above the first half's: its weight is exactly one,
# so that a value met by that key alone comes out as the correctly rounded 1 / (1 + (keys - 1) 2^-x).  Rounding that weight as well adds
# up to half a unit in the last place.  128 CTAs: steps of 128 keys; 512: of 64.
@pytest.mark.parametrize("B", [1, 4])
@pytest.mark.parametrize("dtype,ulp", [(torch.bfloat16, 2.0 ** -7), (torch.float16, 2.0 ** -10)])
@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("rerope", [False, True])
def test_prefill_largest_weight_is_one(api, B, dtype, ulp, D, rerope):
    H, L = 64, 256
    q1 = torch.zeros(B, H, L, D, device="cuda", dtype=dtype)
    q1[..., 0] = 1
    k1 = torch.zeros(B, H, L, D, device="cuda", dtype=dtype)
    k1[:, :, 100, 0] = torch.linspace(1.0, 7.9, B * H, device="cuda").view(B, H).to(dtype)
    v = torch.zeros_like(k1)
    v[:, :, 100] = 1
    scale = 1 / 1.4426950408889634
    q2, k3 = (q1.clone(), k1.clone()) if rerope else (q1, k1)
    out = api.prefill_from_aggregates(q1, q2, k1, k3, v, None, None, None, 256, scale=scale)
    api.check_status()
    for row in (127, 255):
        want = 1 / (1 + row * torch.exp2(-k1[:, :, 100, 0].double()))
        err = (out[:, :, row].double() / want[..., None] - 1).abs().max()
        assert err <= 0.5 * ulp * (1 + 2.0 ** -8) + 1e-6, float(err / ulp)   # half a unit at the bottom of a binade; sums and exponentials are fp32
