"""Cases that the framework's speed is measured on: what programs ask of the sparse-attention path.

``listed()`` names the cases, ``draw(rng)`` gives one more of the same ranges, ``prepare(case, seed)`` makes what a
program holds before the call, ``run(state)`` is one pass through the public entry points, ``work(case)`` the bytes and
operations a pass cannot do without, ``tolerance(case)`` how far the outputs of another correct implementation at the
same precision may lie apart, and ``exact(case, seed)`` the outputs in 64 bits.

Kinds of case (all tensors bf16 [B, H, L, D]; a (batch, head) unit is one attention problem):

* ``layer``  one self-attention call of a layer in next-scale generation: the QKV prologue (normalise, scale, RoPE,
  append to the KV cache), then the attention that the per-(scale, layer) dispatch picks.  ``route`` is ``dense``
  (scales below the decision scale), ``full`` (the decision step: attention, column sums, top-k, O-cache), ``sparse``
  (remapped key lists and the O-cache resized into column-sparse attention) or ``csla`` (static sink + window mask).
* ``mask``   importance scoring for a block mask: attention with exact column sums, then always-kept blocks and the
  top blocks by score.
* ``block``  attention under such a mask, 128x128 or 64x64 blocks.
* ``given``  the ``torch.ops.chipmunk`` operator: attention and column sums from supplied row normalisers.
* ``group``  the operators at another query-group size (192 rows: the geometry of code written for the Triton
  kernels): attention with statistics, column sums per group, top-k, column-sparse attention.
* ``score``  per-scale KV scoring without an attention output: column sums and the best tenth of the keys per head.
* ``evict``  KV-cache compaction of one layer: window scores, pooling, selection, gather.
"""
import math

import torch

import lvar_b200.torch_ops  # noqa: F401  (registers torch.ops.chipmunk)
from lvar_b200 import kernels as K
from lvar_b200 import policy as P
from lvar_b200.infinity_loop import rope2d_tables
from lvar_b200.scalekv import ScaleKVCluster

SCALES = P.INFINITY_SCALES           # sides of the 13 token maps of a 1024 x 1024 image
CUM = P.cumulative_tokens(SCALES)    # start of each scale on the KV axis; CUM[-1] = 10521 tokens
DECISION = 10                        # the 40 x 40 scale
CSLA_WINDOWS = [-1] * 8 + [1, 1, 3, 5, 7]
CSLA_SINK = 5
GROUP, MULTIPLE = 256, 128           # rows per key list, list lengths in multiples of


def listed():
    return [
        # The smallest calls: an early scale of one image (conditional + unconditional copy), 8 x 8 queries on 121 keys.
        # 9 of the 13 scales are like this, once per layer: what counts is the latency of the two launches.
        {"name": "layer dense 8x8", "kind": "layer", "route": "dense", "B": 2, "H": 16, "D": 128, "Lq": 64, "start": 57},
        # The largest scale below the decision scale, one image.
        {"name": "layer dense 32x32", "kind": "layer", "route": "dense", "B": 2, "H": 16, "D": 128, "Lq": 1024, "start": 1497},
        # The decision step of a column-sparse layer, one image.
        {"name": "layer full 40x40", "kind": "layer", "route": "full", "B": 2, "H": 16, "D": 128, "scale": 10},
        # A sparse step of such a layer at the last scale, one image.
        {"name": "layer sparse 64x64", "kind": "layer", "route": "sparse", "B": 2, "H": 16, "D": 128, "scale": 12},
        # Static-mask attention at the last scale for a batch of four images: what two thirds of the layers run at the
        # three largest scales.
        {"name": "layer csla 64x64 B8", "kind": "layer", "route": "csla", "B": 8, "H": 16, "D": 128, "scale": 12},
        # Scoring and selection of the block-sparse benchmark: 64 x 64 queries, all keys, 17 of 83 blocks kept.
        {"name": "mask 64x64", "kind": "mask", "B": 2, "H": 16, "D": 128, "Lq": 4096, "Lkv": 10521, "keep": 17, "sink": 521},
        # The benchmark's headline: block-sparse attention under that mask.
        {"name": "block 64x64", "kind": "block", "B": 2, "H": 16, "D": 128, "Lq": 4096, "Lkv": 10521, "keep": 17,
         "sink": 521, "block": 128},
        # The last scale of a 2048 x 2048 image, 32 heads, 19 of 192 blocks: the largest call.
        {"name": "block 128x128 H32", "kind": "block", "B": 2, "H": 32, "D": 128, "Lq": 16384, "Lkv": 24576, "keep": 19,
         "sink": 0, "block": 128},
        # A 256 x 256 class-conditional model (head dimension 64): last scale, 16 x 16 queries on 680 keys, 64 x 64 blocks.
        {"name": "block 16x16 D64", "kind": "block", "B": 2, "H": 16, "D": 64, "Lq": 256, "Lkv": 680, "keep": 6,
         "sink": 204, "block": 64},
        # The operator form with supplied normalisers, sizes off every tile grid.
        {"name": "given 1000x2999", "kind": "given", "B": 1, "H": 16, "D": 128, "Lq": 1000, "Lkv": 2999},
        # KV scoring over the whole 13-scale schedule of one image, 10 % of the keys kept per head.
        {"name": "score 13 scales", "kind": "score", "B": 2, "H": 16, "D": 128, "first": 0, "last": 12},
        # Compaction of a layer's cache after the 48 x 48 scale: 6425 keys to 2000.
        {"name": "evict 48x48", "kind": "evict", "B": 2, "H": 16, "D": 128, "scale": 11, "keep": 2000},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


#: Dense-equivalent operations that a drawn case may ask for (the largest listed case has 1.3e12).
_MOST = 1.25e12


def draw(rng):
    while True:
        kind = rng.choice(["layer", "layer", "layer", "layer", "mask", "block", "block", "given", "group", "score", "evict"])
        D = 64 if rng.random() < 0.2 else 128
        H = rng.choice([8, 12, 16, 16, 16, 20, 30])
        B = rng.choice([1, 2, 2, 2, 4, 8, 16, 32])
        c = {"kind": kind, "B": B, "H": H, "D": D}
        if kind == "layer":
            route = c["route"] = rng.choice(["dense", "full", "sparse", "csla"])
            if route == "dense":
                c["Lq"] = _log_int(rng, 1, 4096)
                c["start"] = int(c["Lq"] * rng.uniform(0.8, 2.2))
            elif route == "full":
                c["scale"] = DECISION
            elif route == "sparse":
                c["scale"] = rng.choice([11, 12])
            else:
                c["scale"] = rng.choice([10, 11, 12])
        elif kind in ("mask", "block"):
            b = c["block"] = 64 if kind == "block" and rng.random() < 0.3 else 128
            c["Lq"] = _log_int(rng, 200, 16384)
            c["Lkv"] = min(32768, int(c["Lq"] * rng.uniform(1.0, 2.8)))
            nk = -(-c["Lkv"] // b)
            c["keep"] = max(1, min(nk, round(nk * rng.uniform(0.08, 0.4))))
            c["sink"] = rng.choice([0, 0, min(521, c["Lkv"] // 8)])
        elif kind in ("given", "group"):
            c["Lq"] = _log_int(rng, 200, 4096)
            c["Lkv"] = int(c["Lq"] * rng.uniform(1.0, 2.8))
            if kind == "group":
                c["rows"] = 192
                c["keep"] = 64 * max(1, round(c["Lkv"] * rng.uniform(0.04, 0.2) / 64))
        elif kind == "score":
            c["first"] = rng.randrange(0, 13)
            c["last"] = rng.randrange(c["first"], 13)
        else:
            c["scale"] = rng.choice([9, 10, 11, 12])
            c["keep"] = int(CUM[c["scale"] + 1] * rng.uniform(0.05, 0.6))
        known = [{k: v for k, v in x.items() if k != "name"} for x in listed()]
        if c not in known and work(c)["flops"] <= _MOST and B * H <= 275 and _grown(c) <= 3e9:
            return c


def _grown(c):
    """Largest fp32 / int32 array of a pass, in bytes (column sums or key lists)."""
    units = c["B"] * c["H"]
    if c["kind"] in ("mask", "given", "group"):
        return 4.0 * units * c["Lkv"] * -(-c["Lq"] // 128)
    if c["kind"] == "layer" and c["route"] in ("full", "sparse"):
        return 4.0 * units * CUM[c["scale"] + 1] * -(-SCALES[c["scale"]] ** 2 // GROUP)
    return 0.0


# ----------------------------------------------------------------------------------------------- inputs
_BASIS_RANK = 8


def _structured(gen, B, H, L, D, basis, amount):
    """N(0,1) plus a part that lies in a few directions shared by the queries and keys of a head, as attention
    activations have: a few keys matter to most queries, so that column sums spread over several binades."""
    x = torch.randn(B, H, L, D, generator=gen, device="cuda")
    if amount:
        x += amount * (torch.randn(B, H, L, _BASIS_RANK, generator=gen, device="cuda") @ basis)
    return x.bfloat16()


def _qkv(gen, B, H, Lq, Lkv, D):
    basis = torch.randn(1, H, _BASIS_RANK, D, generator=gen, device="cuda")
    q = _structured(gen, B, H, Lq, D, basis, 0.5 * _BASIS_RANK ** -0.5)
    k = _structured(gen, B, H, Lkv, D, basis, 2.0 * _BASIS_RANK ** -0.5)
    v = torch.randn(B, H, Lkv, D, generator=gen, device="cuda").bfloat16()
    return q, k, v


def _random_keys(gen, B, H, G, n, count):
    """count distinct keys of [0, n) per group, in random order."""
    return torch.rand(B, H, G, n, generator=gen, device="cuda").topk(count, dim=-1).indices.to(torch.int32)


def _layer_sizes(c):
    if "scale" in c:
        return SCALES[c["scale"]] ** 2, CUM[c["scale"]]
    return c["Lq"], c["start"]


def _prepare_layer(c, gen):
    B, H, D = c["B"], c["H"], c["D"]
    Lq, start = _layer_sizes(c)
    Lkv = start + Lq
    basis = torch.randn(1, H, _BASIS_RANK, D, generator=gen, device="cuda")

    def rows(L, amount):
        return _structured(gen, B, H, L, D, basis, amount)
    qkv = torch.stack([rows(Lq, 1.0), rows(Lq, 1.0), rows(Lq, 0.0)], 2)       # [B, H, 3, Lq, D]
    cap = max(CUM[-1], Lkv)
    k_cache = torch.zeros(B, H, cap, D, dtype=torch.bfloat16, device="cuda")
    v_cache = torch.zeros_like(k_cache)
    k_cache[:, :, :start] = torch.nn.functional.normalize(rows(start, 1.0).float(), dim=-1).bfloat16()
    v_cache[:, :, :start] = rows(start, 0.0)
    cos, sin = _tables(D)
    s = {"kind": "layer", "route": c["route"], "qkv": qkv.permute(0, 3, 2, 1, 4).contiguous(),     # [B, Lq, 3, H, D]
         "k_cache": k_cache, "v_cache": v_cache, "start": start, "end": Lkv, "cos": cos, "sin": sin,
         "scale_mul": torch.full((H,), 4.0, device="cuda"), "scale_ind": c.get("scale", 0), "spattn": None, "before": None,
         "layer_ind": 20 if c["route"] == "csla" else 0}
    layer = s["layer"] = P.SelfAttentionDispatch(s["layer_ind"], None, SCALES, scale=1.0)
    if c["route"] == "csla":
        s["spattn"] = P.SparseFlexAttn([(x, x) for x in SCALES], CSLA_WINDOWS, c["scale"], CSLA_SINK, num_heads=H)
    if c["route"] == "sparse":
        # what the scales before left in the layer's storage: the decision scale's keys, and after the 48 x 48 scale
        # also that scale's own band; the previous scale's O-cache
        prev = c["scale"] - 1
        n_src, groups = CUM[prev + 1], -(-SCALES[prev] ** 2 // GROUP)
        top = P.indices_count(0.05, CUM[DECISION + 1], MULTIPLE)
        lists = torch.zeros(B, H, groups, n_src, dtype=torch.int32, device="cuda")
        lists[..., :top] = _random_keys(gen, B, H, groups, CUM[DECISION + 1], top)
        count = top
        if prev > DECISION:
            band, n_band = P.local_band(SCALES, prev, 7, GROUP, MULTIPLE)
            lists[..., top:top + n_band] = band.to(device="cuda", dtype=torch.int32)
            count += n_band
        counts = torch.full((B, H, groups), count, dtype=torch.int32, device="cuda")
        cache = (0.3 * torch.randn(B, H, SCALES[prev] ** 2, D, generator=gen, device="cuda")).bfloat16()
        s["before"] = (lists, counts, count, cache)
    s["store"] = layer.sparse_attn.storage
    return s


_TABLES = {}


def _tables(D):
    """RoPE tables of the model, shared by all layers and images (longer sequences than the schedule's repeat them)."""
    if D not in _TABLES:
        cos, sin = rope2d_tables(SCALES, D, device="cuda")
        _TABLES[D] = (torch.cat([cos, cos]), torch.cat([sin, sin]))
    return _TABLES[D]


def _recipe_mask(gen, c):
    """Always-kept blocks and, per (batch, head, row), the best others of random scores."""
    B, H, Lq, Lkv, b = c["B"], c["H"], c["Lq"], c["Lkv"], c.get("block", 128)
    nq, nk = -(-Lq // b), -(-Lkv // b)
    always = P.sink_local_blocks(nq, nk, b, c["sink"], Lkv - Lq, 0, Lq).cuda()
    scores = torch.rand(B, H, nq, nk, generator=gen, device="cuda") + 2.0 * always
    pick = scores.topk(max(c["keep"], 1), dim=-1).indices
    mask = torch.zeros(B, H, nq, nk, dtype=torch.bool, device="cuda").scatter_(-1, pick, True)
    return mask | always


def prepare(case, seed):
    c = case
    gen = torch.Generator(device="cuda").manual_seed(seed)
    kind, B, H, D = c["kind"], c["B"], c["H"], c["D"]
    if kind == "layer":
        return _prepare_layer(c, gen)
    s = {"kind": kind, "case": c, "scale": D ** -0.5}
    if kind == "score":
        basis = torch.randn(1, H, _BASIS_RANK, D, generator=gen, device="cuda")
        s["k"] = _structured(gen, B, H, CUM[c["last"] + 1], D, basis, 2.0 * _BASIS_RANK ** -0.5)
        s["q"] = {i: _structured(gen, B, H, SCALES[i] ** 2, D, basis, 0.5 * _BASIS_RANK ** -0.5)
                  for i in range(c["first"], c["last"] + 1)}
        return s
    if kind == "evict":
        Lq, Lkv = SCALES[c["scale"]] ** 2, CUM[c["scale"] + 1]
        s["q"], s["k"], s["v"] = _qkv(gen, B, H, Lq, Lkv, D)
        # every layer's budget after this scale; the window is one token of each patch of a 4 x 4 grid
        s["cluster"] = ScaleKVCluster([[c["keep"]]] * len(SCALES), window_size=16, base_capacity=121)
        return s
    s["q"], s["k"], s["v"] = _qkv(gen, B, H, c["Lq"], c["Lkv"], D)
    if kind == "mask":
        nq, nk = -(-c["Lq"] // 128), -(-c["Lkv"] // 128)
        s["always"] = P.sink_local_blocks(nq, nk, 128, c["sink"], c["Lkv"] - c["Lq"], 0, c["Lq"]).cuda()
    elif kind == "block":
        s["mask"] = _recipe_mask(gen, c)
    elif kind == "given":
        # row normalisers of an earlier pass: 1 / sum_j exp(s_ij)
        p = torch.empty(B, H, c["Lq"], 1, device="cuda")
        for b in range(B):
            for h in range(H):
                p[b, h, :, 0] = torch.exp(-torch.logsumexp(s["q"][b, h].float() @ s["k"][b, h].float().T * s["scale"], -1))
        s["p"] = p
    elif kind == "group":
        s["o"] = (0.3 * torch.randn(B, H, c["Lq"], D, generator=gen, device="cuda")).bfloat16()
    return s


# ----------------------------------------------------------------------------------------------- one pass
def _run_layer(s):
    st = s["store"]
    if s["before"] is not None:  # every image comes to this scale with what the scales before left
        st.indices, st.counts, st.count_value, st.out_cache = s["before"]
    a, b = s["start"], s["end"]
    q = K.qkv_prologue(s["qkv"], s["scale_mul"], s["cos"], s["sin"], a, s["k_cache"], s["v_cache"], a)
    o = s["layer"](q, s["k_cache"][:, :, :b], s["v_cache"][:, :, :b], scale_ind=s["scale_ind"], layer_ind=s["layer_ind"],
                   spattn_fn=s["spattn"])
    out = {"o": o, "q": q, "k": s["k_cache"][:, :, a:b], "v": s["v_cache"][:, :, a:b]}
    if s["route"] == "full":
        out.update(lists=st.indices, counts=st.counts, cache=st.out_cache)
    elif s["route"] == "sparse":
        out.update(lists=st.indices, counts=st.counts)
    return out


def run(state):
    s = state
    kind = s["kind"]
    if kind == "layer":
        return _run_layer(s)
    c = s["case"]
    if kind == "mask":
        o, cs = K.dense_colsum_attn_fwd(s["q"], s["k"], s["v"], s["scale"])
        return {"o": o, "cs": cs, "mask": K.block_mask_from_colsums(cs, s["always"], c["keep"], 128)}
    if kind == "block":
        return K.block_sparse_attn_fwd(s["q"], s["k"], s["v"], s["mask"], s["scale"], block=c["block"])
    if kind == "given":
        return torch.ops.chipmunk.dense_colsum_attn_scaled(s["q"], s["k"], s["v"], s["p"], s["scale"])
    if kind == "group":
        o, M, L = K.dense_attn_fwd(s["q"], s["k"], s["v"], s["scale"])
        cs = K.colsum_groups_fwd(s["q"], s["k"], M, L, c["rows"], s["scale"])
        lists, counts = K.topk_indices(cs, c["keep"], out_cols=c["Lkv"], with_counts=True)
        out = K.csp_attn_fwd(s["q"], s["k"], s["v"], lists, counts, s["o"], 1, c["rows"], s["scale"])
        return {"o": o, "M": M, "L": L, "cs": cs, "lists": lists, "counts": counts, "out": out}
    if kind == "score":
        out = []
        for i, q in s["q"].items():
            n = CUM[i + 1]
            row = K.colsum_tiles_fwd(q, s["k"][:, :, :n], s["scale"]).sum(dim=2, keepdim=True)
            keep = round(0.1 * n)
            out.append((row, K.topk_indices(row, keep, ascending_index=True)) if keep else (row,))
        return out
    if kind == "evict":
        return s["cluster"].update_kv(s["k"], s["q"], s["v"], c["scale"])
    raise ValueError(kind)


# ----------------------------------------------------------------------------------------------- work and tolerance
def work(case):
    """Every input read once, every output written once; 4 D operations per attended (query, key) pair (scores and
    weighted sum), 2 D where only the scores are taken."""
    c = case
    kind, B, H, D = c["kind"], c["B"], c["H"], c["D"]
    U = B * H
    if kind == "layer":
        Lq, start = _layer_sizes(c)
        Lkv = start + Lq
        # qkv in, q and o out, new cache rows out, old cache rows in
        by = 2.0 * U * D * (3 * Lq + 2 * Lq + 2 * Lq + 2 * start)
        pairs = float(Lq) * Lkv
        if c["route"] == "full":
            G, top = -(-Lq // GROUP), P.indices_count(0.05, Lkv, MULTIPLE)
            pairs += float(Lq) * top
            by += 2.0 * U * D * Lq + 4.0 * U * G * (Lkv + 1)
        elif c["route"] == "sparse":
            prev = c["scale"] - 1
            G, n = -(-Lq // GROUP), {11: 896, 12: 1408}[c["scale"]]
            pairs = float(Lq) * n
            by += 2.0 * U * D * SCALES[prev] ** 2 + 4.0 * U * (-(-SCALES[prev] ** 2 // GROUP)) * 256 + 4.0 * U * G * (Lkv + 1)
        elif c["route"] == "csla":
            m = _csla_mask(c["scale"])
            pairs = _active_pairs(m, Lq, Lkv, 128)
        return {"bytes": by, "flops": 4.0 * D * U * pairs}
    if kind == "score":
        by = fl = 0.0
        for i in range(c["first"], c["last"] + 1):
            Lq, Lkv = SCALES[i] ** 2, CUM[i + 1]
            by += U * (2.0 * D * (Lq + Lkv) + 4.0 * Lkv + 4.0 * round(0.1 * Lkv))
            fl += 2.0 * D * U * Lq * Lkv
        return {"bytes": by, "flops": fl}
    if kind == "evict":
        Lkv = CUM[c["scale"] + 1]
        return {"bytes": U * (2.0 * D * (Lkv + c["keep"]) + 2.0 * D * 2 * c["keep"]), "flops": 2.0 * D * U * 16 * Lkv}
    Lq, Lkv = c["Lq"], c["Lkv"]
    by = 2.0 * U * D * (2 * Lq + 2 * Lkv)
    pairs = float(Lq) * Lkv
    if kind == "mask":
        nq, nk = -(-Lq // 128), -(-Lkv // 128)
        by += 4.0 * U * nq * Lkv + U * nq * nk
    elif kind == "block":
        b = c["block"]
        nq, nk = -(-Lq // b), -(-Lkv // b)
        by += U * nq * nk
        always = P.sink_local_blocks(nq, nk, b, c["sink"], Lkv - Lq, 0, Lq).sum(-1)
        pairs = float(always.clamp(min=c["keep"]).sum()) * b * b
    elif kind == "given":
        by += 4.0 * U * (2 * Lq + -(-Lq // GROUP) * Lkv)
    elif kind == "group":
        G = -(-Lq // c["rows"])
        by += 2.0 * U * D * 2 * Lq + 4.0 * U * (2 * Lq + G * (2 * Lkv + 1))
        pairs += float(Lq) * c["keep"]
    return {"bytes": by, "flops": 4.0 * D * U * pairs}


_MASKS = {}


def _csla_mask(scale):
    if scale not in _MASKS:
        _MASKS[scale] = P.csla_block_mask([(x, x) for x in SCALES], CSLA_WINDOWS, scale, CSLA_SINK, 128)
    return _MASKS[scale]


def _active_pairs(mask, Lq, Lkv, b):
    nq, nk = mask.shape
    rows = torch.full((nq,), float(b))
    cols = torch.full((nk,), float(b))
    rows[-1], cols[-1] = Lq - (nq - 1) * b, Lkv - (nk - 1) * b
    return float((mask.float() * rows.view(-1, 1) * cols.view(1, -1)).sum())


def tolerance(case):
    kind = case["kind"]
    if kind == "score":
        # fp32 sums of fp32 exponentials: 1e-7 to 4e-7 (single values 1.5e-6) from fp64 with hardware exponentials, up to
        # 2.7e-6 where they come from a polynomial
        return {"rel": 1e-5, "max": 6e-5, "differ": 0.01}
    if kind == "evict":
        # a selection by bf16-rounded logits: the rounding points are part of the operation
        return "exact"
    # bf16 outputs of sums over bf16-rounded probabilities: 2.1e-3 to 2.3e-3 (single values 1.1e-2) from fp64
    tol = {"rel": 1e-2, "max": 0.05, "differ": 0.005}
    if kind == "group" or case.get("route") == "full":
        # two keys whose column sums agree to the last bits may change places, at the end of a list for good: the
        # rows that attend it then differ by that key's share
        tol["max"] = 0.3
    return tol


# ----------------------------------------------------------------------------------------------- the same in 64 bits
def _probabilities(q, k, scale, keep=None):
    """Softmax rows of one (batch, head) unit in fp64, with the row maxima and sums of the scores; ``keep``: a mask."""
    s = (q.double() @ k.double().T) * scale
    if keep is not None:
        s.masked_fill_(~keep, float("-inf"))
    m = s.max(-1, keepdim=True).values
    s.sub_(m).exp_()
    n = s.sum(-1, keepdim=True)
    return s.div_(n), m, n


def _by_group(p, rows):
    """Sums over groups of ``rows`` query rows."""
    pad = -p.shape[0] % rows
    return torch.nn.functional.pad(p, (0, 0, 0, pad)).view(-1, rows, p.shape[1]).sum(1)


def _listed_attention(q, k, v, scale, lists, rows):
    """Attention of each group of ``rows`` query rows over the keys of its list, fp64."""
    out = []
    for g in range(lists.shape[0]):
        i = lists[g].long()
        out.append(_probabilities(q[g * rows:(g + 1) * rows], k[i], scale)[0] @ v[i].double())
    return torch.cat(out)


def _units(fn, B, H):
    """fn(b, h) gives a tuple of tensors of one unit; stacked to [B, H, ...]."""
    got = [[fn(b, h) for h in range(H)] for b in range(B)]
    return [torch.stack([torch.stack([got[b][h][i] for h in range(H)]) for b in range(B)]) for i in range(len(got[0][0]))]


def _exact_layer(c, s):
    B, H = c["B"], c["H"]
    a, e = s["start"], s["end"]
    q, k, v = (s["qkv"][:, :, i].permute(0, 2, 1, 3).double() for i in range(3))
    cos, sin = s["cos"][a:e].double(), s["sin"][a:e].double()

    def turn(x):
        x = x / x.norm(dim=-1, keepdim=True)
        x0, x1 = x[..., 0::2], x[..., 1::2]
        return torch.stack([cos * x0 - sin * x1, sin * x0 + cos * x1], -1).flatten(-2)
    q, k = turn(q) * s["scale_mul"].double().view(1, H, 1, 1), turn(k)
    out = {"q": q, "k": k, "v": v}
    # the attention reads what the prologue stores, which is bf16
    Q = q.bfloat16()
    Kc = torch.cat([s["k_cache"][:, :, :a], k.bfloat16()], 2)
    V = torch.cat([s["v_cache"][:, :, :a], v.bfloat16()], 2)
    route, rows = c["route"], GROUP
    if route == "dense":
        out["o"], = _units(lambda b, h: (_probabilities(Q[b, h], Kc[b, h], 1.0)[0] @ V[b, h].double(),), B, H)
    elif route == "csla":
        m = _csla_mask(c["scale"]).cuda().repeat_interleave(128, 0).repeat_interleave(128, 1)[:e - a, :e]
        out["o"], = _units(lambda b, h: (_probabilities(Q[b, h], Kc[b, h], 1.0, m)[0] @ V[b, h].double(),), B, H)
    elif route == "full":
        top = P.indices_count(0.05, e, MULTIPLE)

        def unit(b, h):
            p = _probabilities(Q[b, h], Kc[b, h], 1.0)[0]
            o = p @ V[b, h].double()
            lists = _by_group(p, rows).topk(top, -1).indices
            return o, o - _listed_attention(Q[b, h], Kc[b, h], V[b, h], 1.0, lists, rows)
        out["o"], out["cache"] = _units(unit, B, H)
        out.update(lists=None, counts=None)
    else:
        lists, _, count, cache = s["before"]
        band = s["layer"].sparse_attn.local_inds[c["scale"]][0].cuda()
        Gk, Gs = band.shape[0], lists.shape[2]
        near = ((torch.arange(Gk).float() + 0.5) / Gk * Gs - 0.5).round().long().clamp(0, Gs - 1)
        side, prev = SCALES[c["scale"]], SCALES[c["scale"] - 1]

        def unit(b, h):
            mine = torch.cat([lists[b, h, near.cuda(), :count], band], -1)
            grid = cache[b, h].double().view(prev, prev, -1).permute(2, 0, 1)[None]
            grid = torch.nn.functional.interpolate(grid, size=(side, side), mode="bilinear", align_corners=False)
            return grid[0].flatten(1).T + _listed_attention(Q[b, h], Kc[b, h], V[b, h], 1.0, mine, rows),
        out["o"], = _units(unit, B, H)
        out.update(lists=None, counts=None)
    return out


def exact(case, seed):
    """What ``run`` returns for these inputs, in fp64 by plain torch; ``None`` for selections and for ``evict``, whose
    outputs are copies of inputs chosen by bf16-rounded scores."""
    c = case
    kind, B, H = c["kind"], c["B"], c["H"]
    if kind == "evict":
        return None
    s = prepare(c, seed)
    if kind == "layer":
        return _exact_layer(c, s)
    if kind == "score":
        sc = s["scale"]
        out = []
        for i, q in s["q"].items():
            n = CUM[i + 1]
            row, = _units(lambda b, h: (_probabilities(q[b, h], s["k"][b, h, :n], sc)[0].sum(0, keepdim=True),), B, H)
            out.append((row, None) if round(0.1 * n) else (row,))
        return out
    q, k, v, sc = s["q"], s["k"], s["v"], s["scale"]
    if kind == "mask":
        def unit(b, h):
            p = _probabilities(q[b, h], k[b, h], sc)[0]
            return p @ v[b, h].double(), _by_group(p, 128)
        o, cs = _units(unit, B, H)
        return {"o": o, "cs": cs, "mask": None}
    if kind == "block":
        def unit(b, h):
            m = s["mask"][b, h].repeat_interleave(c["block"], 0).repeat_interleave(c["block"], 1)[:c["Lq"], :c["Lkv"]]
            return _probabilities(q[b, h], k[b, h], sc, m)[0] @ v[b, h].double(),
        return _units(unit, B, H)[0]
    if kind == "given":
        def unit(b, h):
            p, m, n = _probabilities(q[b, h], k[b, h], sc)
            total = m.exp() * n
            return p @ v[b, h].double(), _by_group(p * (total * s["p"][b, h].double()), GROUP), 1 / total
        return _units(unit, B, H)
    if kind == "group":
        def unit(b, h):
            p, m, n = _probabilities(q[b, h], k[b, h], sc)
            o, cs = p @ v[b, h].double(), _by_group(p, c["rows"])
            lists = cs.topk(c["keep"], -1).indices
            return (o, m[:, 0] * math.log2(math.e), n[:, 0], cs,
                    s["o"][b, h].double() + _listed_attention(q[b, h], k[b, h], v[b, h], sc, lists, c["rows"]))
        o, M, L, cs, out = _units(unit, B, H)
        return {"o": o, "M": M, "L": L, "cs": cs, "lists": None, "counts": None, "out": out}
    raise ValueError(kind)
