"""A wait limit of zero in every form of the attention kernel: the launch gives up at its first unfinished wait, returns with
a status word, and leaves the device, the work counter and the next call as they were.

Nothing faults here: a wait that runs out ends in an ordinary return."""
import pytest
import torch

pytestmark = pytest.mark.gpu

B, H, ROWS = 2, 3, 256
# many tiles a block, and calls whose copies are all under way before anything waits for them
SIZES = [(600, 1500), (60, 200)]


def _qkv(D, LQ, LKV):
    gen = torch.Generator(device="cuda").manual_seed(D)
    return [torch.randn(B, H, n, D, generator=gen, device="cuda").bfloat16() for n in (LQ, LKV, LKV)]


def _copy_only(x):
    """The values of x with batches that are not whole rows apart: no 2-D tensor of rows, so rows are copied."""
    b, h, L, D = x.shape
    y = torch.empty(b * (h * L * D + 8), device=x.device, dtype=x.dtype).as_strided(x.shape, (h * L * D + 8, L * D, D, 1))
    return y.copy_(x)


def _lists(G, LKV):
    """Whole runs of consecutive keys, scattered tiles between them and a short last tile."""
    gen = torch.Generator(device="cuda").manual_seed(3)
    idx = torch.arange(LKV, device="cuda", dtype=torch.int32).expand(B, H, G, LKV).clone()
    for at in (128, 512, 768):
        if at + 128 > LKV:
            break
        idx[..., at:at + 128] = torch.randint(0, LKV, (B, H, G, 128), generator=gen, device="cuda", dtype=torch.int32)
    return idx, torch.full((B, H, G), min(1100, LKV), dtype=torch.int32, device="cuda")


def _csp(layout):
    def call(K, D, size, status):
        q, k, v = _qkv(D, *size)
        if layout == "copies":
            k, v = _copy_only(k), _copy_only(v)
        idx, counts = _lists(-(-size[0] // ROWS), size[1])
        return (K.csp_attn_fwd(q, k, v, idx, counts, torch.zeros_like(q), 1, ROWS, status=status),)
    return call


def _block(K, D, size, status):
    q, k, v = _qkv(D, *size)
    mask = (torch.arange(-(-size[1] // 128), device="cuda") + torch.arange(-(-size[0] // 128), device="cuda")[:, None]) % 3 != 2
    return (K.block_sparse_attn_fwd(q, k, v, mask, status=status),)


def _sums(form):
    def call(K, D, size, status):
        q, k, v = _qkv(D, *size)
        if form == "two sweeps":
            return K.dense_colsum_attn_fwd(q, k, v, return_stats=True, status=status)
        if form == "no output":
            return K.colsum_tiles_fwd(q, k, return_stats=True, status=status)
        M, L = (torch.full((B, H, size[0]), x, device="cuda") for x in (2.0, 300.0))
        if form == "given, no output":
            return (K.colsum_tiles_fwd(q, k, stats=(M, L), status=status),)
        return K.dense_colsum_attn_given_fwd(q, k, v, M, L, return_stats=True, status=status)
    return call


def _dense(K, D, size, status):
    return K.dense_attn_fwd(*_qkv(D, *size), status=status)


def _stand_alone(K, D, size, status):
    q, k, _ = _qkv(D, *size)
    M, L = (torch.full((B, H, size[0]), x, device="cuda") for x in (2.0, 300.0))
    return (K.colsum_fwd(q, k, M, L, 192, status=status),)


CALLS = {"dense": _dense, "csp rows": _csp("rows"), "csp copies": _csp("copies"), "block": _block}
CALLS["sums, stand-alone"] = _stand_alone
CALLS |= {f"sums, {form}": _sums(form) for form in ("two sweeps", "no output", "given, no output", "given")}


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("size", SIZES)
@pytest.mark.parametrize("form", list(CALLS))
def test_wait_limit_zero_returns_a_status_and_the_next_call_is_right(form, size, D, monkeypatch):
    from lvar_b200 import _lib
    from lvar_b200 import kernels as K
    call = CALLS[form]
    good = K.new_status("cuda")
    want = call(K, D, size, good)
    for _ in range(3):
        given_up = K.new_status("cuda")
        with monkeypatch.context() as m:
            m.setattr(_lib, "DEFAULT_WAIT_NS", 0)
            call(K, D, size, given_up)
        assert K.read_status(given_up)[0] == 6
        assert all(torch.equal(a, b) for a, b in zip(call(K, D, size, good), want))
    assert K.read_status(good)[0] == 0
