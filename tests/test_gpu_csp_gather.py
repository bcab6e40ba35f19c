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


def _case(B, H, D, count, kind="mixed", Lq=600, L=1500, rows=256):
    gen = torch.Generator(device="cuda").manual_seed(D + count)
    q, k, v, o = (torch.randn(B, H, n, D, generator=gen, device="cuda").bfloat16() for n in (Lq, L, L, Lq))
    G = -(-Lq // rows)
    idx = _lists(kind, B, H, G, L, gen)
    return q, k, v, o, idx, torch.full((B, H, G), count, dtype=torch.int32, device="cuda"), rows


def _gathered(rows_view, *tensors):
    return all(rows_view(t.shape, t.stride()) is not None for t in tensors)


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("kind", ["scattered", "runs", "mixed"])
def test_the_two_routes_are_two_and_match_the_oracle(rows_view, D, kind):
    from lvar_b200 import kernels as K
    from oracle import attention as oa
    q, k, v, o, idx, counts, rows = _case(2, 3, D, 1000, kind)
    ks, vs = _layouts(k), _layouts(v)
    for name in ks:
        assert _gathered(rows_view, ks[name], vs[name]) == (name != "copies"), name
    ref = oa.csp_attn(*(t.cpu() for t in (q, k, v)), None, idx.cpu(), counts.cpu(), o.cpu(), 1, bm=rows).float()
    for name in ("copies", "contiguous"):
        d = (K.csp_attn_fwd(q, ks[name], vs[name], idx, counts, o, 1, rows).float().cpu() - ref).abs()
        # delta within 2e-2 and the sum rounded to bf16 once more: an ulp of 4 to 8 is 3.1e-2
        assert d.max().item() <= 3.2e-2 and d.mean().item() <= 2e-3, name


@pytest.mark.parametrize("D", [64, 128])
def test_one_tensor_that_cannot_be_gathered_sends_both_to_copies(rows_view, D):
    from lvar_b200 import kernels as K
    q, k, v, o, idx, counts, rows = _case(2, 3, D, 1000)
    ks, vs = _layouts(k), _layouts(v)
    want = K.csp_attn_fwd(q, ks["copies"], vs["copies"], idx, counts, o, 1, rows)
    for a, b in [("copies", "contiguous"), ("cache", "copies"), ("heads in a row", "cache"), ("contiguous", "side by side")]:
        assert _gathered(rows_view, ks[a], vs[b]) == ("copies" not in (a, b))
        assert torch.equal(K.csp_attn_fwd(q, ks[a], vs[b], idx, counts, o, 1, rows), want), (a, b)


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("B,H", [(1, 3), (2, 1), (1, 1)])
def test_strides_of_a_single_batch_or_head_do_not_matter(rows_view, B, H, D):
    from lvar_b200 import kernels as K
    q, k, v, o, idx, counts, rows = _case(B, H, D, 1000)
    L = k.shape[2]

    def odd(x):   # the stride of an extent of one is off the rows
        sb, sh = (24 if B == 1 else H * L * D), (40 if H == 1 else L * D)
        return torch.empty(B * H * L * D, device="cuda", dtype=x.dtype).as_strided(x.shape, (sb, sh, D, 1)).copy_(x)
    want = K.csp_attn_fwd(q, k, v, idx, counts, o, 1, rows)
    ko, vo = odd(k), odd(v)
    assert _gathered(rows_view, ko, vo)
    assert torch.equal(K.csp_attn_fwd(q, ko, vo, idx, counts, o, 1, rows), want)


@pytest.mark.parametrize("layout", ["contiguous", "copies"])
@pytest.mark.parametrize("D", [64, 128])
def test_an_index_out_of_range_is_reported_and_reads_key_0(layout, D):
    from lvar_b200 import kernels as K
    q, k, v, o, idx, counts, rows = _case(2, 3, D, 1000, "scattered")
    k, v = _layouts(k)[layout], _layouts(v)[layout]
    bad, zero = idx.clone(), idx.clone()
    for at, value in [(5, k.shape[2]), (300, -1), (999, 2 ** 31 - 1)]:
        bad[1, 2, 1, at], zero[1, 2, 1, at] = value, 0
    status, clean = K.new_status("cuda"), K.new_status("cuda")
    got = K.csp_attn_fwd(q, k, v, bad, counts, o, 1, rows, status=status)
    assert torch.equal(got, K.csp_attn_fwd(q, k, v, zero, counts, o, 1, rows, status=clean))
    assert K.read_status(status)[0] == 5 and K.read_status(clean)[0] == 0
