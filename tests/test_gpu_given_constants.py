"""Attention and column sums from supplied statistics: constants that are not finite stay what they are, also where the last KV
tile is short and its missing columns are masked."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("Lq,Lkv", [(200, 512), (200, 500), (128, 129), (1500, 1300)])
def test_an_infinite_constant_gives_infinite_statistics(D, Lq, Lkv):
    """M = -inf with L > 0 is the constant +inf: every probability of the row is infinite, so its returned L is."""
    from lvar_b200 import kernels as K
    gen = torch.Generator(device="cuda").manual_seed(Lkv)
    q, k, v = (torch.randn(1, 2, n, D, generator=gen, device="cuda").bfloat16() for n in (Lq, Lkv, Lkv))
    _, M, L = K.dense_attn_fwd(q, k, v)
    o, cs, Mo, Lo = K.dense_colsum_attn_given_fwd(q, k, v, M, L, return_stats=True)
    rows = [0, 77, Lq - 1]
    Mi = M.clone()
    Mi[:, 1, rows] = -float("inf")
    o2, cs2, Mo2, Lo2 = K.dense_colsum_attn_given_fwd(q, k, v, Mi, L, return_stats=True)
    assert torch.isposinf(Lo2[:, 1, rows]).all() and torch.isneginf(Mo2[:, 1, rows]).all()
    assert torch.isnan(o2[:, 1, rows].float()).all()
    keep = torch.ones(2, Lq, dtype=torch.bool)
    keep[1, rows] = False
    for a, b in ((o, o2), (Mo, Mo2), (Lo, Lo2)):
        assert torch.equal(a[0][keep], b[0][keep])
    tiles = sorted({r // 128 for r in rows})
    assert torch.isposinf(cs2[0, 1, tiles]).all() and torch.equal(cs[0, 0], cs2[0, 0])


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("Lkv", [512, 500])
def test_a_nan_constant_stays_nan(D, Lkv):
    from lvar_b200 import kernels as K
    gen = torch.Generator(device="cuda").manual_seed(Lkv)
    q, k, v = (torch.randn(1, 1, n, D, generator=gen, device="cuda").bfloat16() for n in (200, Lkv, Lkv))
    _, M, L = K.dense_attn_fwd(q, k, v)
    M[0, 0, 3] = float("nan")
    o, cs, _, Lo = K.dense_colsum_attn_given_fwd(q, k, v, M, L, return_stats=True)
    assert torch.isnan(Lo[0, 0, 3]) and torch.isnan(o[0, 0, 3].float()).all() and torch.isnan(cs[0, 0, 0]).all()
    assert torch.isfinite(Lo[0, 0, 4:]).all() and torch.isfinite(cs[0, 0, 1]).all()
