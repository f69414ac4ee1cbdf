"""GPU tests of the branches that a call's type, size or alignment selects, at the sizes where each can go wrong."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def api():
    from vqtree_b200 import api as _api
    return _api


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _rn(g, *s):
    return torch.randn(*s, generator=g, device="cuda")


# rows gathered as 16-byte vectors (64, 128, 256, 512 bytes a row; the first falls back to single elements), indexes outside the array
@pytest.mark.parametrize("dtype,D", [(torch.bfloat16, 32), (torch.bfloat16, 64), (torch.float16, 128), (torch.float32, 128)])
@pytest.mark.parametrize("idx", [torch.int64, torch.int32])
def test_gather_aggregates_moves_whole_rows(api, dtype, D, idx):
    g = _gen(D)
    B, H, L, NB, C = 2, 3, 300, 3, 131
    v = _rn(g, B, H, L + 1, D).to(dtype)
    vi = torch.randint(-2, L + 4, (B, H, NB + 1, C), generator=g, device="cuda").to(idx)
    cnt = torch.randint(0, 3, (B, H, NB, C), generator=g, device="cuda").float()
    for c in (None, cnt):
        got = api.gather_aggregates(v, vi, NB, c)
        at = vi[:, :, :NB].long()
        ok = (at >= 0) & (at <= L) & (torch.ones_like(cnt, dtype=torch.bool) if c is None else c > 0)
        want = torch.gather(v, 2, at.clamp(0, L).reshape(B, H, -1, 1).expand(-1, -1, -1, D)).reshape(B, H, NB, C, D)
        assert torch.equal(got, torch.where(ok[..., None], want, torch.zeros_like(want)))
