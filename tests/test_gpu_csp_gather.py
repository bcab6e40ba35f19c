"""Column-sparse attention: the TMA row gather against the cp.async gather, over the layouts that choose between them.

Which one runs depends on the strides alone: K and V rows come by TMA where a tensor is one 2-D tensor of rows (batches
whole rows apart, heads whole rows apart or side by side in a row), by cp.async otherwise.  Both put the same bytes into
the same tiles, so the outputs are equal bit for bit."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _layouts(x):
    """The values of x [B, H, L, D] in the layouts under test, the copy-only one first."""
    B, H, L, D = x.shape
    odd = torch.empty(B * (H * L * D + 8), device=x.device, dtype=x.dtype)
    odd = odd.as_strided((B, H, L, D), (H * L * D + 8, L * D, D, 1))   # batches not whole rows apart
    odd.copy_(x)
    cache = torch.zeros(B, H, L + 37, D, device=x.device, dtype=x.dtype)
    cache[:, :, :L] = x
    packed = torch.zeros(B, L, 3, H, D, device=x.device, dtype=x.dtype)
    packed[:, :, 1] = x.permute(0, 2, 1, 3)
    return {"copies": odd, "contiguous": x.contiguous(), "cache": cache[:, :, :L],
            "heads in a row": packed[:, :, 1].permute(0, 2, 1, 3),
            "side by side": x.permute(0, 2, 1, 3).contiguous().permute(0, 2, 1, 3)}


def _lists(kind, B, H, G, L, gen):
    if kind == "scattered":
        return torch.rand(B, H, G, L, generator=gen, device="cuda").argsort(-1).int()
    run = torch.arange(L, device="cuda", dtype=torch.int32).expand(B, H, G, L).clone()
    if kind == "runs":          # many tiles in a row that no gather warp but one is needed for
        return run
    mixed = run
    mixed[..., 128:256] = torch.randint(0, L, (B, H, G, 128), generator=gen, device="cuda", dtype=torch.int32)
    mixed[..., 640:700] = mixed[..., 640:700].flip(-1)
    return mixed


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("kind", ["scattered", "runs", "mixed"])
@pytest.mark.parametrize("count", [0, 1, 128, 129, 1000, 1500])
def test_tma_gather_gives_the_bits_of_the_copies(D, kind, count):
    from lvar_b200 import kernels as K
    B, H, Lq, L, rows = 2, 3, 600, 1500, 256
    gen = torch.Generator(device="cuda").manual_seed(D + count)
    q, k, v, o = (torch.randn(B, H, n, D, generator=gen, device="cuda").bfloat16() for n in (Lq, L, L, Lq))
    G = -(-Lq // rows)
    idx = _lists(kind, B, H, G, L, gen)
    counts = torch.full((B, H, G), count, dtype=torch.int32, device="cuda")
    counts[0, 1, 1] = count // 2
    status = K.new_status("cuda")
    ks, vs = _layouts(k), _layouts(v)
    want = K.csp_attn_fwd(q, ks["copies"], vs["copies"], idx, counts, o, 1, rows, status=status)
    assert torch.isfinite(want.float()).all()
    for name in ks:
        got = K.csp_attn_fwd(q, ks[name], vs[name], idx, counts, o, 1, rows, status=status)
        assert torch.equal(got, want), name
    assert K.read_status(status)[0] == 0
