"""Performance cases of SparseConv2D: what a user of this package has it do, call by call.

A case is one call, or one training step, of the public surface on one GPU:

  infer    y = layer(x, table)                                       an adapter at inference
  train    y = layer(x, table); gradients of x, weight and bias      an adapter in a training step
  step     scores -> build_neighbor_table -> the training step       the layer right after a selection
  table    scores -> build_neighbor_table                            token selection alone
  rounds   full-grid table, then select_and_update per round         the pruning schedule of a backbone

Values follow the benchmark configurations of this repository: features and upstream gradients N(0,1),
Kaiming-normal weights, kept tokens as the top-k of N(0,1) scores, per slice or per clip.

Keys of a case
  clips, slices, h, w   token grid: `clips` batch rows of `slices` slices of h x w tokens
  keep                  kept share of a segment (1.0: the full grid, every token and its neighbours)
  per_clip              top-k over a whole clip (the reference backbone) instead of over each slice
  cin, cout, ksize      layer
  dtype                 activations; `amp`: fp32 parameters under bf16 autocast (mixed-precision training)
  table                 "built": by this package; "given": a table the caller made (plain tensor, batch-global
                        indices); "local": a caller's table with indices local to each clip
"""
import math

import torch

import eccv26_tad_b200 as svtad

DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16, "fp32": torch.float32}
ELEM = {"bf16": 2, "fp16": 2, "fp32": 4}


def _case(name, kind, **kw):
    c = dict(kind=kind, clips=1, slices=8, h=14, w=14, keep=0.3, per_clip=False, cin=192, cout=192, ksize=3,
             dtype="bf16", amp=False, table="built")
    c.update(kw)
    if name is not None:
        c["name"] = name
    return c


def listed():
    return [
        # one short clip through an fp32 layer: the smallest call (784 rows), all latency
        _case("infer_fp32_784_rows", "infer", slices=8, keep=0.5, dtype="fp32"),
        # one clip on a 16 x 16 grid, 16 slices, keep 0.7 over the clip: 2868 rows (ragged), half precision serving
        _case("infer_fp16_one_clip", "infer", slices=16, h=16, w=16, keep=0.7, per_clip=True, cin=256, cout=256,
              dtype="fp16"),
        # an adapter in front of the first selection: the full 14 x 14 grid of 24 short clips (37 632 rows)
        _case("infer_bf16_full_grid", "infer", clips=24, slices=8, keep=1.0, cin=128, cout=128),
        # mixed precision on a table the caller's own code made, late in a three-round schedule: 24 x 339 rows
        _case("train_amp_given_table", "train", clips=24, slices=8, keep=0.216, per_clip=True, cin=128, cout=128,
              amp=True, table="given"),
        # the benchmark's layer at its largest keep rate (17 280 rows) ...
        _case("train_bf16_keep55", "train", clips=2, slices=80, keep=0.55),
        # ... and at its smallest with a new table every step: selection, table and the layer behind them (3 200 rows)
        _case("step_bf16_keep10", "step", clips=2, slices=80, keep=0.10),
        # embedding width 384 with a 4x bottleneck: a channel count that is no multiple of 64
        _case("train_bf16_width96", "train", clips=2, slices=80, keep=0.3, cin=96, cout=96),
        # full precision training
        _case("train_fp32", "train", clips=1, slices=80, keep=0.3, dtype="fp32"),
        # large layers: 18 880 rows
        _case("train_bf16_c256_5x5", "train", clips=4, slices=80, keep=0.3, cin=256, cout=256, ksize=5),
        _case("train_bf16_c1024", "train", clips=4, slices=80, keep=0.3, cin=1024, cout=1024),
        # selection alone, 3 072 slices in one call, and the three-round schedule of two 160-frame clips
        _case("table_3072_slices", "table", clips=8, slices=384, keep=0.25),
        _case("rounds_two_long_clips", "rounds", clips=2, slices=80, keep=0.6, per_clip=True),
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


#: most work of a drawn layer, in rows * taps * cin * cout: the large 16-bit layer above, and the fp32 one (also for
#: 16-bit layers whose channel counts are no multiples of 64); of the wide one's products a third are there at keep 0.3
MOST_WIDE = 18880 * 9 * 1024 * 1024
MOST_NARROW = 4720 * 9 * 192 * 192


def draw(rng):
    kind = rng.choices(["train", "infer", "step", "table", "rounds"], [9, 5, 2, 2, 2])[0]
    h, w = rng.choice([(14, 14), (14, 14), (10, 10), (16, 16), (11, 13)])
    if kind == "table":
        return _case(None, kind, clips=rng.choice([1, 2, 8]), slices=_log_uniform(rng, 8, 384), h=h, w=w,
                     keep=round(rng.uniform(0.1, 0.7), 3), ksize=rng.choice([3, 3, 3, 5]))
    if kind == "rounds":
        return _case(None, kind, clips=rng.choice([1, 2, 4, 8, 24]), slices=_log_uniform(rng, 8, 80), h=h, w=w,
                     keep=round(rng.uniform(0.5, 0.8), 3), per_clip=True)
    while True:
        dtype = rng.choices(["bf16", "fp16", "fp32"], [6, 2, 2])[0]
        cin = rng.choice([64, 96, 128, 192, 256, 320, 384, 512, 768, 1024])
        cout = cin if rng.random() < 0.8 else rng.choice([64, 96, 128, 192, 256])
        c = _case(None, kind, clips=rng.choice([1, 1, 2, 4, 8, 24]), slices=_log_uniform(rng, 4, 160), h=h, w=w,
                  keep=1.0 if rng.random() < 0.1 else round(rng.uniform(0.1, 0.7), 3), per_clip=rng.random() < 0.4,
                  cin=cin, cout=cout, ksize=rng.choice([3, 3, 3, 3, 5]), dtype=dtype,
                  amp=kind == "train" and dtype == "bf16" and rng.random() < 0.4,
                  table="built" if kind == "step" else rng.choices(["built", "given", "local"], [7, 2, 1])[0])
        dense = _rows(c) * c["ksize"] ** 2 * cin * cout
        most = MOST_WIDE if dtype != "fp32" and cin % 64 == 0 and cout % 64 == 0 else MOST_NARROW
        if dense <= most and 3 * _pairs(c) * cin * cout <= MOST_WIDE and _rows(c) <= 80000:
            return c


def _segments(c):
    """(segments, tokens of a segment, kept tokens of a segment)"""
    hw = c["h"] * c["w"]
    n_seg, seg_len = (c["clips"], c["slices"] * hw) if c["per_clip"] else (c["clips"] * c["slices"], hw)
    return n_seg, seg_len, svtad.num_keep_tokens(c["keep"], seg_len)


def _rows(c):
    n_seg, _, k = _segments(c)
    return n_seg * k


def _round_sizes(c):
    sizes = [c["slices"] * c["h"] * c["w"]]
    for _ in range(3):
        sizes.append(svtad.num_keep_tokens(c["keep"], sizes[-1]))
    return sizes


class State:
    pass


def prepare(case, seed):
    c, s = case, State()
    s.case = c
    dev = torch.device("cuda")
    g = torch.Generator(device=dev)
    g.manual_seed(int(seed) * 2654435761 % (1 << 62) + 17)

    def normal(*shape):
        return torch.randn(*shape, generator=g, device=dev, dtype=torch.float32)

    if c["kind"] == "rounds":
        s.scores = [normal(c["clips"], n) for n in _round_sizes(c)[:3]]
        return s
    n_seg, seg_len, k = _segments(c)
    s.scores = normal(n_seg, seg_len)
    if c["kind"] == "table":
        return s

    dtype = DTYPES[c["dtype"]]
    n, kk = n_seg * k, c["ksize"] ** 2
    if c["kind"] != "step":
        if c["keep"] == 1.0:
            table = svtad.get_initial_neighbor_indices(c["h"], c["w"], c["slices"], dev, c["clips"], c["ksize"])
        else:
            table = svtad.build_neighbor_table(s.scores, None, c["h"], c["w"], c["ksize"], num_keep=k)[1]
        if c["table"] != "built":
            table = table.reshape(c["clips"], n // c["clips"], kk).clone()
        if c["table"] == "local":
            first = torch.arange(c["clips"], device=dev, dtype=torch.int32).view(-1, 1, 1) * (n // c["clips"])
            table = torch.where(table >= 0, table - first, table)
        s.table = table
    layer = svtad.SparseConv2d(c["cin"], c["cout"], kernel_size=c["ksize"]).to(dev)
    with torch.no_grad():
        layer.weight.copy_(normal(kk, c["cin"], c["cout"]) * math.sqrt(2.0 / (c["cin"] * kk)))
        layer.bias.copy_(normal(c["cout"]) * 0.1)
    s.layer = layer if c["amp"] else layer.to(dtype)
    s.x = normal(c["clips"], n // c["clips"], c["cin"]).to(dtype)
    if c["kind"] == "infer":
        s.layer.eval()
        return s
    s.x.requires_grad_(True)
    s.gy = normal(c["clips"], n // c["clips"], c["cout"]).to(dtype)
    return s


def _train(s, table):
    if s.case["amp"]:
        with torch.autocast("cuda", dtype=torch.bfloat16):
            y = s.layer(s.x, table)
    else:
        y = s.layer(s.x, table)
    gx, gw, gb = torch.autograd.grad(y, (s.x, s.layer.weight, s.layer.bias), s.gy)
    return {"y": y.detach(), "grad_x": gx, "grad_weight": gw, "grad_bias": gb}


def run(s):
    c = s.case
    if c["kind"] == "infer":
        with torch.no_grad():
            return s.layer(s.x, s.table)
    if c["kind"] == "train":
        return _train(s, s.table)
    if c["kind"] == "rounds":
        table = svtad.get_initial_neighbor_indices(c["h"], c["w"], c["slices"], "cuda", c["clips"], c["ksize"])
        out = []
        for r, k in enumerate(_round_sizes(c)[1:]):
            idx, table = svtad.select_and_update(s.scores[r], table, k)
            out += [idx, table]
        return out
    kept, table = svtad.build_neighbor_table(s.scores, None, c["h"], c["w"], c["ksize"], num_keep=_segments(c)[2])
    if c["kind"] == "table":
        return {"kept": kept, "table": table}
    return dict(_train(s, table), kept=kept, table=table)


def _pairs(c):
    """Expected (row, tap) pairs whose neighbour is kept: the products the layer cannot do without."""
    n_seg, seg_len, k = _segments(c)
    h, w, r = c["h"], c["w"], c["ksize"] // 2
    other = (k - 1) / (seg_len - 1) if seg_len > 1 else 0.0
    inside = sum(max(0, h - abs(dy)) * max(0, w - abs(dx)) / (h * w)
                 for dy in range(-r, r + 1) for dx in range(-r, r + 1) if (dy, dx) != (0, 0))
    return n_seg * k * (1.0 + inside * other)


def work(case):
    c = case
    kk = c["ksize"] ** 2
    if c["kind"] == "rounds":
        sizes, b = _round_sizes(c), c["clips"]
        # full-grid table written; per round the scores and the kept rows read, indices (int64) and new rows written
        moved = 4 * sizes[0] * kk + sum(4 * p + 4 * n * kk + 8 * n + 4 * n * kk for p, n in zip(sizes, sizes[1:]))
        return {"bytes": b * moved, "flops": 0}
    n_seg, seg_len, k = _segments(c)
    n = n_seg * k
    table = 4 * n_seg * seg_len + 4 * n + 4 * n * kk
    if c["kind"] == "table":
        return {"bytes": table, "flops": 0}
    e, p = ELEM[c["dtype"]], 4 if c["amp"] else ELEM[c["dtype"]]
    params = (kk * c["cin"] * c["cout"] + c["cout"]) * p
    flops = 2.0 * _pairs(c) * c["cin"] * c["cout"]
    if c["kind"] == "infer":
        return {"bytes": n * (c["cin"] + c["cout"]) * e + 4 * n * kk + params, "flops": flops}
    moved = 2 * n * (c["cin"] + c["cout"]) * e + 2 * params + (table if c["kind"] == "step" else 4 * n * kk)
    return {"bytes": moved, "flops": 3 * flops}


def tolerance(case):
    if case["kind"] in ("table", "rounds"):
        return "exact"
    # one rounding of the result to the activations' type on top of 32-bit sums; tables are exact
    return {"rel": {"bf16": 1e-2, "fp16": 2e-3, "fp32": 1e-5}[case["dtype"]]}
