"""ScaleKV compaction on the GPU against the CPU oracle and the reference's golden selections."""
import pytest
import torch

pytestmark = pytest.mark.gpu

from test_scalekv_oracle import _case, tie_aware_equal  # noqa: E402


@pytest.fixture(scope="module")
def K():
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    from lvar_b200 import kernels
    return kernels


@pytest.mark.parametrize("name", ["c", "d"])
def test_scores_pool_and_selection_match_oracle(K, golden_scalekv, name):
    from oracle import scalekv as osk
    scale_ind, cap, pooling, q, k, v, window, want = _case(golden_scalekv, name)
    key_len, Lq = k.shape[2], q.shape[2]
    wdev = torch.tensor(window, dtype=torch.int32, device="cuda")
    scores = K.scalekv_scores(q.cuda(), k.cuda(), wdev, key_len - Lq)
    ref = osk.window_scores(q, k, window).float()
    got = scores.cpu()
    assert torch.equal(torch.isinf(got), torch.isinf(ref))
    fin = torch.isfinite(ref)
    # bf16 values: identical up to a rare flip of the last bf16 bit (fp32 summation order inside a dot product)
    assert (got[fin] - ref[fin]).abs().max().item() <= 2.0 ** -7 * ref[fin].abs().max().item()
    assert (got[fin] == ref[fin]).float().mean().item() > 0.97
    for pool in ("maxpool", "avgpool"):
        pooled = K.scalekv_pool(scores, wdev, 5, pool).cpu()
        pref = osk.pooled_scores(scores.cpu().to(torch.bfloat16), 5, pool).float()
        pref[..., window] = float("inf")
        assert torch.equal(pooled, pref)
    # the whole selection, against the oracle's pooled scores (ties and last-bit flips may swap keys)
    pooled = K.scalekv_pool(scores, wdev, 5, pooling)
    idx = K.topk_indices(pooled, cap, ascending_index=True).cpu()
    _, opooled = osk.select_indices(q, k, window, cap, 5, pooling)
    for h in range(2):
        assert torch.equal(idx[0, h], torch.sort(idx[0, h]).values) and len(set(idx[0, h].tolist())) == cap
        assert set(window) <= set(idx[0, h].tolist())
        assert tie_aware_equal(idx[0, h], want[0, h], opooled[0, h].float(), slack=2.0 ** -6)


def test_cluster_update_kv_end_to_end(K, golden_scalekv):
    from lvar_b200.scalekv import ScaleKVCluster
    scale_ind, cap, pooling, q, k, v, window, want = _case(golden_scalekv, "d")
    c = ScaleKVCluster([[cap] * 4 for _ in range(16)], window_size=16, base_capacity=121, kernel_size=5,
                       pooling=pooling, layer_idx=1)
    qd, kd, vd = q.cuda(), k.cuda(), v.cuda()
    ko, vo = c.update_kv(kd, qd, vd, scale_ind)
    assert ko.shape == (1, 2, cap, k.shape[-1]) and vo.shape == ko.shape and c.max_capacity == cap
    idx = c.select_indices(kd, qd, scale_ind).cpu().long()
    for h in range(2):
        assert torch.equal(ko[0, h].cpu(), k[0, h][idx[0, h]]) and torch.equal(vo[0, h].cpu(), v[0, h][idx[0, h]])
    # below the base capacity, and when the cache already fits its budget, nothing is touched
    c2 = ScaleKVCluster([[5000] * 4 for _ in range(16)], layer_idx=0)
    k_small = kd[:, :, :100]
    assert c2.update_kv(k_small, qd[:, :, :100], vd[:, :, :100], 3)[0] is k_small
    assert c2.update_kv(kd, qd, vd, scale_ind)[0] is kd


def test_gather_rows_strided_and_clamped(K):
    g = torch.Generator().manual_seed(2)
    big = torch.randn(2, 3, 50, 3 * 64, generator=g).bfloat16().cuda()
    src = big[..., 64:128]                      # a strided view with a contiguous last dimension
    idx = torch.randint(-3, 60, (2, 3, 17), generator=g, dtype=torch.int32).cuda()
    out = K.gather_rows(src, idx)
    ref = torch.gather(src, 2, idx.clamp(0, 49).long().unsqueeze(-1).expand(-1, -1, -1, 64))
    assert torch.equal(out, ref)


def test_scalekv_argument_errors(K):
    q = torch.zeros(1, 1, 16, 64, dtype=torch.bfloat16, device="cuda")
    w = torch.arange(70, dtype=torch.int32, device="cuda")
    with pytest.raises(RuntimeError, match="window"):
        K.scalekv_scores(q, q, w, 0)
    with pytest.raises(RuntimeError, match="bfloat16"):
        K.scalekv_scores(q.float(), q, w[:4], 0)


@pytest.mark.parametrize("D,Lkv,w", [(128, 1, 1), (128, 128, 16), (128, 129, 7), (128, 6425, 16), (64, 127, 8), (64, 700, 64),
                                     (128, 300, 64), (64, 257, 9)])
def test_scores_bits_follow_the_stated_order(K, D, Lkv, w):
    """The order of a logit's sum is fixed: D/8 sums of 8 consecutive products, then pairs p and p + D/16, p + D/32, ...
    Products of bf16 numbers are exact in fp32, so plain fp32 arithmetic restates it bit for bit."""
    g = torch.Generator().manual_seed(Lkv + w)
    B, H, Lq = 1, 3, max(w, min(Lkv, 100))
    q = torch.randn(B, H, Lq, D, generator=g).bfloat16().cuda()
    kbig = torch.randn(B, H, Lkv, 2 * D, generator=g).bfloat16().cuda()
    k = kbig[..., D:]                                    # rows of a wider buffer
    window = torch.randperm(max(Lkv, w), generator=g)[:w].sort().values.to(torch.int32).cuda()
    offset = Lkv - Lq
    got = K.scalekv_scores(q, k, window, offset)
    wq = q[:, :, (window.long() - offset).clamp(0, Lq - 1)].float()
    prod = (wq.unsqueeze(3) * k.float().unsqueeze(2)).view(B, H, w, Lkv, D // 8, 8)
    part = torch.zeros_like(prod[..., 0])
    for e in range(8):
        part = part + prod[..., e]
    while part.shape[-1] > 1:
        half = part.shape[-1] // 2
        part = part[..., :half] + part[..., half:]
    logit = (part[..., 0].bfloat16().float() / torch.tensor(float(D)).sqrt().cuda()).bfloat16().float()
    total = torch.zeros(B, H, Lkv, device="cuda")
    for i in range(w):
        total = total + logit[:, :, i]
    total = total.bfloat16().float()
    inside = window[window < Lkv].long()
    total[..., inside] = float("-inf")
    assert torch.equal(got, total)


def test_window_only_selection_is_the_callers_own(K):
    """With a budget of the window alone the returned indices are a fresh tensor, not the shared window, and several
    scales and repeated calls keep their own windows."""
    from lvar_b200.scalekv import ScaleKVCluster, window_indices
    q = torch.randn(1, 1, 1600, 64).bfloat16().cuda()
    for _ in range(2):
        for lq, lkv, scale in ((1600, 4121, 10), (1024, 2521, 9), (1600, 4121, 10)):
            c = ScaleKVCluster([[16]] * 13, window_size=16)
            c.max_capacity = 16
            k = torch.randn(1, 1, lkv, 64).bfloat16().cuda()
            idx = c.select_indices(k, q[:, :, :lq], scale)
            assert idx[0, 0].tolist() == window_indices(lq, lkv - lq, lkv, 16)
            idx.fill_(-1)


@pytest.mark.parametrize("B,H,L,n,D", [(1, 1, 1, 1, 8), (2, 3, 70, 129, 128), (1, 2, 40, 33, 24), (1, 1, 9, 5, 2056), (3, 5, 200, 64, 64),
                                       (2, 40000, 3, 2, 8)])
def test_gather_rows_shapes(K, B, H, L, n, D):
    """Rows shorter and longer than a block's pieces, piece counts that do not divide it, counts off the rows a thread
    takes, more (batch, head) pairs than a grid row count allows, indices out of range on both sides."""
    g = torch.Generator().manual_seed(n)
    src = torch.randn(B, H, L, D, generator=g).bfloat16().cuda()
    idx = torch.randint(-2, L + 2, (B, H, n), generator=g, dtype=torch.int32).cuda()
    want = torch.gather(src, 2, idx.clamp(0, L - 1).long().unsqueeze(-1).expand(-1, -1, -1, D))
    assert torch.equal(K.gather_rows(src, idx), want)


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("w,Lkv", [(1, 300), (4, 129), (16, 130), (9, 17), (64, 200), (6, 1000), (7, 1000)])
def test_scores_of_few_and_many_keys_are_the_same_bits(K, D, w, Lkv):
    """One head by itself (shared keys where the rule says few) and as one of enough heads that the rule says many."""
    g = torch.Generator().manual_seed(w * Lkv)
    copies = 73 + 9000 * 8 // Lkv * 8 // min(w, 8)
    q = torch.randn(1, 1, max(w, 8), D, generator=g).bfloat16().cuda()
    k = torch.randn(1, 1, Lkv, D, generator=g).bfloat16().cuda()
    window = torch.randperm(max(Lkv, w), generator=g)[:w].sort().values.to(torch.int32).cuda()
    one = K.scalekv_scores(q, k, window, 3)
    many = K.scalekv_scores(q.expand(1, copies, -1, -1), k.expand(1, copies, -1, -1), window, 3)
    assert torch.equal(many, one.expand_as(many))


@pytest.mark.parametrize("B,H,L,n,D", [(2, 150, 20, 63, 128), (2, 150, 20, 65, 128), (1, 293, 5, 129, 64), (1, 300, 7, 1, 24), (2, 147, 3, 5, 2056)])
def test_gather_rows_four_per_thread(K, B, H, L, n, D):
    """Enough blocks for four rows per thread: counts below, at and off a block's share."""
    test_gather_rows_shapes(K, B, H, L, n, D)
