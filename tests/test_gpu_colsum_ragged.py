"""Column sums of a last query tile with few rows: the sweep leaves out the 32-row chunks that hold none."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("rows", [1, 31, 32, 33, 64, 65, 96, 97, 127, 128])
def test_sums_of_a_ragged_tile_match_the_oracle(rows, D):
    from lvar_b200 import kernels as K
    from oracle import attention as oa
    B, H, Lq, Lkv = 1, 2, 256 + rows, 700
    gen = torch.Generator().manual_seed(rows)
    q, k, v = (torch.randn(B, H, n, D, generator=gen).bfloat16() for n in (Lq, Lkv, Lkv))
    _, ref = oa.dense_colsum_attn(q, k, v, None, 128, dtype=torch.float64)
    qc, kc, vc = q.cuda(), k.cuda(), v.cuda()
    status = K.new_status("cuda")
    cs, M, L = K.colsum_tiles_fwd(qc, kc, return_stats=True, status=status)
    for got in (cs, K.colsum_tiles_fwd(qc, kc, stats=(M, L), status=status),
                K.dense_colsum_attn_fwd(qc, kc, vc, status=status)[1]):
        assert got.shape == ref.shape
        # element-wise, fp32 sums of at most 128 probabilities against 64 bits: the 1e-3 bar of the sums
        assert ((got.double().cpu() - ref.double()).abs() / ref.double()).max().item() <= 1e-3
    assert K.read_status(status)[0] == 0
