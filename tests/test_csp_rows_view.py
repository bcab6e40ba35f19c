"""Which K and V tensors column-sparse attention gathers by TMA: the rule against plain stride arithmetic, on the host.

A tensor that the rule accepts is addressed as rows of pitch sl; every element must lie where its strides say, inside the rows and
columns that the tensor map names, and those must not reach past the tensor's own last element."""
import itertools
import random

import torch


def _check(view, shape, strides):
    B, H, L, D = shape
    sb, sh, sl = strides[:3]
    rb, rh, ch, rows, width = view
    assert width <= sl and rows < 2 ** 31 and width < 2 ** 31
    last = sum((n - 1) * s for n, s in zip((B, H, L), (sb, sh, sl))) + D - 1
    assert (rows - 1) * sl + width - 1 == last
    for b, h, l, d in itertools.product((0, B - 1), (0, H // 2, H - 1), (0, L // 2, L - 1), (0, D - 1)):
        row, col = b * rb + h * rh + l, h * ch + d
        assert row < rows and col < width
        assert row * sl + col == b * sb + h * sh + l * sl + d
        assert (h * ch * 2) % 16 == 0          # where a request starts in its row


def _layouts(B, H, L, D):
    """name -> (tensor, whether rows are gathered by TMA)"""
    def new(*shape):
        return torch.empty(*shape, dtype=torch.bfloat16, device="meta")

    def strided(*strides):
        return new(2 ** 33).as_strided((B, H, L, D), strides)
    x, cache, packed = new(B, H, L, D), new(B, H, L + 37, D), new(B, L, 3, H, D)
    return {
        "contiguous": (x, True),
        "slice of a cache": (cache[:, :, :L], True),
        "middle of a cache": (cache[:, :, 5:5 + L], True),
        "side by side": (new(B, L, H, D).permute(0, 2, 1, 3), True),
        "packed qkv": (packed[:, :, 1].permute(0, 2, 1, 3), True),
        "heads first": (new(H, B, L, D).permute(1, 0, 2, 3), True),
        "batches off the rows": (strided(H * L * D + 8, L * D, D, 1), B == 1),
        "heads off the rows": (strided(H * (L * D + 8), L * D + 8, D, 1), H == 1 and B == 1),
        "rows that overlap": (strided(H * L * D, L * D, D - 8, 1), False),
    }


def test_layouts_and_their_route(rows_view):
    for B, H, L, D in [(2, 3, 1500, 64), (2, 3, 1500, 128), (1, 3, 77, 128), (2, 1, 77, 64), (1, 1, 1, 128), (16, 16, 10521, 128)]:
        for name, (t, gathered) in _layouts(B, H, L, D).items():
            view = rows_view(t.shape, t.stride())
            assert (view is not None) == gathered, (name, t.shape, t.stride())
            if view:
                _check(view, t.shape, t.stride())


def test_strides_of_extents_of_one_do_not_matter(rows_view):
    for D in (64, 128):
        assert rows_view((1, 4, 100, D), (8, 100 * D, D)) is not None       # any batch stride
        assert rows_view((4, 1, 100, D), (100 * D, 8, D)) is not None       # any head stride
        assert rows_view((1, 1, 100, D), (8, 24, D)) is not None


def test_random_strides(rows_view):
    rng = random.Random(0)
    accepted = 0
    for _ in range(20000):
        D = rng.choice([64, 128])
        shape = (rng.choice([1, 2, 5]), rng.choice([1, 2, 7]), rng.choice([1, 2, 100, 1500]), D)
        sl = rng.choice([D, D, 2 * D, 7 * D, D + 8, 8 * rng.randrange(0, 300)])
        sh = rng.choice([0, D, sl, shape[2] * sl, (shape[2] + 3) * sl, 8 * rng.randrange(0, 4000)])
        sb = rng.choice([0, sl, shape[1] * sh, shape[2] * sl, shape[1] * shape[2] * sl, 8 * rng.randrange(0, 100000)])
        view = rows_view(shape, (sb, sh, sl))
        if view:
            accepted += 1
            _check(view, shape, (sb, sh, sl))
        else:
            rows_apart = sl >= D and (shape[0] == 1 or sb % sl == 0)
            heads_ok = shape[1] == 1 or (sl and (sh % sl == 0 or (shape[1] - 1) * sh + D <= sl))
            assert not (rows_apart and heads_ok), (shape, sb, sh, sl)
    assert accepted > 2000


def test_row_numbers_stay_in_32_bits(rows_view):
    """Row and column numbers are 32-bit in a request; tensors beyond that are copied."""
    D = 128
    assert rows_view((2, 1, 100, D), ((2 ** 31 - 101) * D, 0, D)) is not None
    assert rows_view((2, 1, 100, D), ((2 ** 31 - 99) * D, 0, D)) is None
    assert rows_view((1, 2, 100, D), (0, 2 ** 31 * D, D)) is None
    assert rows_view((1, 1, 2, D), (0, 0, 2 ** 39)) is None                 # a pitch of 2^40 bytes
