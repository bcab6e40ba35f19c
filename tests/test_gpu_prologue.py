"""Fused QKV prologue on the GPU against the CPU oracle (itself pinned on the reference's outputs)."""
import pytest
import torch

pytestmark = pytest.mark.gpu

from test_prologue_oracle import SCALES, case  # noqa: E402


@pytest.fixture(scope="module")
def K():
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    from lvar_b200 import kernels
    return kernels


def _close_bf16(got: torch.Tensor, want: torch.Tensor) -> None:
    """Equal except for a rare flip of the last bf16 bit (the fp32 sum of squares is taken in another order)."""
    g, w = got.float().cpu(), want.float()
    assert (g == w).float().mean().item() > 0.999
    assert ((g - w).abs() <= 2.0 ** -7 * w.abs() + 1e-30).all()


@pytest.mark.parametrize("name", ["a", "b"])
def test_prologue_matches_oracle_and_reference(K, golden_prologue, name):
    from oracle import prologue as op
    B, L, H, c, scale_ind, qkv, sm, cos, sin = case(golden_prologue, name)
    start = sum(s * s for s in SCALES[:scale_ind])
    cap, pos = start + L + 5, start
    k_cache = torch.full((B, H, cap, c), 7.0, dtype=torch.bfloat16, device="cuda")
    v_cache = torch.full((B, H, cap, c), 7.0, dtype=torch.bfloat16, device="cuda")
    q = K.qkv_prologue(qkv.cuda(), sm.cuda(), cos.cuda(), sin.cuda(), start, k_cache, v_cache, pos)
    _close_bf16(q, golden_prologue[f"{name}_q_out"])
    _close_bf16(k_cache[:, :, pos:pos + L], golden_prologue[f"{name}_k_out"])
    assert torch.equal(v_cache[:, :, pos:pos + L].cpu(), qkv[:, :, 2].permute(0, 2, 1, 3))
    # rows outside the appended range are untouched
    assert (k_cache[:, :, :pos] == 7).all() and (k_cache[:, :, pos + L:] == 7).all()
    assert (v_cache[:, :, :pos] == 7).all() and (v_cache[:, :, pos + L:] == 7).all()
    # relayout only
    q2 = K.qkv_prologue(qkv.cuda(), None, None, None, 0, k_cache, v_cache, 0)
    oq, ok, _ = op.qkv_prologue(qkv, None, None, None, 0)
    assert torch.equal(q2.cpu(), oq) and torch.equal(k_cache[:, :, :L].cpu(), ok)


def test_prologue_feeds_attention_like_the_reference_call_site(K, golden_prologue):
    """q, the appended K cache and V cache go straight into dense attention: same result as attention on the
    oracle's tensors (the reference casts its fp32 q and k to bf16 at this point)."""
    from oracle import prologue as op
    B, L, H, c, scale_ind, qkv, sm, cos, sin = case(golden_prologue, "b")
    start = sum(s * s for s in SCALES[:scale_ind])
    oq, ok, ov = op.qkv_prologue(qkv, sm, cos, sin, start)
    k_cache = torch.zeros((B, H, L, c), dtype=torch.bfloat16, device="cuda")
    v_cache = torch.zeros_like(k_cache)
    q = K.qkv_prologue(qkv.cuda(), sm.cuda(), cos.cuda(), sin.cuda(), start, k_cache, v_cache, 0)
    o, _, _ = K.dense_attn_fwd(q, k_cache, v_cache, 1.0)
    ref = torch.nn.functional.scaled_dot_product_attention(oq.float(), ok.float(), ov.float(), scale=1.0)
    assert (o.float().cpu() - ref).abs().max().item() <= 2e-2


def test_prologue_argument_errors(K):
    qkv = torch.zeros(1, 4, 3, 2, 64, dtype=torch.bfloat16, device="cuda")
    cache = torch.zeros(1, 2, 3, 64, dtype=torch.bfloat16, device="cuda")
    with pytest.raises(RuntimeError, match="room for rows"):
        K.qkv_prologue(qkv, None, None, None, 0, cache, cache.clone(), 0)
    with pytest.raises(RuntimeError, match="bfloat16"):
        K.qkv_prologue(qkv.float(), None, None, None, 0, cache, cache.clone(), 0)


@pytest.mark.parametrize("B,L,H,c", [(1, 1, 1, 128), (2, 7, 3, 128), (1, 5, 4, 64), (3, 2, 9, 64), (2, 33, 16, 128), (1, 3, 17, 64)])
def test_prologue_8_byte_rows_give_the_same_bits(K, B, L, H, c):
    """Rows on 16-byte boundaries and rows that are only 8-byte aligned, head counts off the warp's share, and rows
    with extreme, infinite and NaN elements: the same bits from both kernels, and those of plain division."""
    g = torch.Generator().manual_seed(B * 1000 + L * 10 + H)
    qkv = torch.randn(B, L, 3, H, c, generator=g).bfloat16()
    qkv[0, 0, 0, 0, 0] = float("inf")
    qkv[0, 0, 1, 0, 1] = float("nan")
    qkv[0, 0, 1, 0, 2] = 3e38
    if L > 1:
        qkv[0, 1, 0, 0, :4] = torch.tensor([3e38, -3e38, 1e-38, 5.0])   # the sum of squares overflows
        qkv[0, 1, 1, 0] *= 1e-25                                         # the norm is clamped
        qkv[0, 1, 1, H - 1] = 0.0
    qkv = qkv.cuda()
    sm = (torch.rand(H, generator=g) * 4).cuda()
    ang = torch.rand(L + 2, c // 2, generator=g) * 6
    cos, sin = ang.cos().cuda(), ang.sin().cuda()

    def caches(shift):
        return [torch.zeros(B * H * (L + 3) * c + 4, dtype=torch.bfloat16, device="cuda")[shift:shift + B * H * (L + 3) * c]
                .view(B, H, L + 3, c) for _ in range(2)]
    k0, v0 = caches(0)
    q0 = K.qkv_prologue(qkv, sm, cos, sin, 2, k0, v0, 3)
    shifted = torch.zeros(qkv.numel() + 4, dtype=torch.bfloat16, device="cuda")[4:].view(qkv.shape)   # 8-byte aligned
    shifted.copy_(qkv)
    k1, v1 = caches(4)
    q1 = K.qkv_prologue(shifted, sm, cos, sin, 2, k1, v1, 3)
    for a, b in ((q0, q1), (k0, k1), (v0, v1)):
        assert torch.equal(a.view(torch.int16), b.view(torch.int16))
    assert torch.equal(v0[:, :, 3:].view(torch.int16), qkv[:, :, 2].permute(0, 2, 1, 3).contiguous().view(torch.int16))

    # the row's sum of squares in the kernel's order: c/32 consecutive squares, then pairs at distance 16, 8, ..., 1
    def unit(x, mul):
        x = x.permute(0, 2, 1, 3).float()
        parts = torch.zeros(x.shape[:-1] + (32,), device="cuda", dtype=torch.float64)
        xd = x.double().view(*x.shape[:-1], 32, c // 32)
        for e in range(c // 32):                       # fp32 fused multiply-add: one rounding of the exact sum
            parts = (parts + xd[..., e] * xd[..., e]).float().double()
        s = parts.float()
        for d in (16, 8, 4, 2, 1):
            s = s[..., :d] + s[..., d:]
        n = s.sqrt()
        n = torch.where(n > 1e-12, n, torch.tensor(1e-12, device="cuda"))
        x = x / n
        if mul is not None:
            x = x * mul.view(1, H, 1, 1)
        x0, x1 = x[..., 0::2], x[..., 1::2]
        cs, sn = cos[2:], sin[2:]
        return torch.stack([cs * x0 - sn * x1, sn * x0 + cs * x1], -1).flatten(-2).bfloat16()
    for got, want in ((q0, unit(qkv[:, :, 0], sm)), (k0[:, :, 3:], unit(qkv[:, :, 1], None))):
        fin = torch.isfinite(want)
        assert torch.equal(torch.isnan(got), torch.isnan(want))
        assert torch.equal(got[fin], want[fin])


@pytest.mark.parametrize("c", [64, 128])
@pytest.mark.parametrize("rope", [False, True])
def test_prologue_division_bits(K, c, rope):
    """Zeros of both signs, subnormal and tiny elements beside large ones, exponents over the whole range: bit for bit
    plain fp32 division, rotation and one rounding to bf16.  The rows' sums of squares are exact here (one large power of
    two, the rest far below its last bit, or rows so small that the norm is clamped), so any order of the sum gives them."""
    g = torch.Generator().manual_seed(c)
    B, L, H = 1, 64, 4
    mant = torch.randint(128, 256, (B, L, 3, H, c), generator=g).float()
    e = torch.randint(-140, -20, (B, L, 3, H, c), generator=g)
    e[:, ::4] = torch.randint(-80, -60, (B, L // 4, 3, H, c), generator=g)
    x = mant.double() * torch.exp2(e.double()) * (1 - 2 * torch.randint(0, 2, mant.shape, generator=g))
    x[..., 0] = torch.exp2(torch.randint(20, 60, x.shape[:-1], generator=g).double())    # the norm
    x[:, 1::4, ..., 0] = 1e-30                                                           # clamped norm, squares underflow
    x[:, 1::4] = x[:, 1::4].clamp(-1e-30, 1e-30)
    x[..., 3], x[..., 10], x[..., 11] = -0.0, 0.0, -0.0
    x[:, 2::4, ..., 16:] = -0.0
    qkv = x.float().bfloat16().cuda()
    sm = torch.tensor([1.0, 0.37, 4.0, 2.5]).cuda()
    ang = torch.rand(L, c // 2, generator=g) * 6
    cos, sin = (ang.cos().cuda(), ang.sin().cuda()) if rope else (None, None)
    kc = torch.zeros(B, H, L, c, dtype=torch.bfloat16, device="cuda")
    vc = torch.zeros_like(kc)
    q = K.qkv_prologue(qkv, sm, cos, sin, 0, kc, vc, 0)

    def unit(y, mul):
        y = y.permute(0, 2, 1, 3).float()
        y = y / y.double().pow(2).sum(-1, keepdim=True).float().sqrt().clamp_min(1e-12)
        if mul is not None:
            y = y * mul.view(1, H, 1, 1)
        if rope:
            y0, y1 = y[..., 0::2], y[..., 1::2]
            y = torch.stack([cos * y0 - sin * y1, sin * y0 + cos * y1], -1).flatten(-2)
        return y.bfloat16()
    for got, want in ((q, unit(qkv[:, :, 0], sm)), (kc, unit(qkv[:, :, 1], None))):
        assert torch.equal(got.view(torch.int16), want.view(torch.int16))


@pytest.mark.parametrize("B,L,H,c", [(2, 7, 1, 128), (3, 3, 1, 64), (1, 5, 2, 64), (2, 130, 2, 128), (1, 1, 1, 64)])
def test_prologue_tokens_that_share_a_warp(K, B, L, H, c):
    """One and two heads: a warp takes several tokens (over the batch), the last warp fewer."""
    test_prologue_8_byte_rows_give_the_same_bits(K, B, L, H, c)
