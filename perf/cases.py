"""The workloads whose speed this framework answers for, as calls of its public entry points.

A case is a dict of plain values.  `kind` names the path:

  stack       EncoderStack.forward: a stack of post-LN encoder layers on a resident batch
  serve       HostPipeline.submit / drain: the same stack fed from and drained to pinned host memory
  ffn-tile    the feed-forward block over packed 16x16 tile-CSR weights (two linear_tile_packed)
  ffn-rowcol  the feed-forward block with pruned hidden units (linear_row, then linear_col)
  1x16, csr   one Linear over 1x16-vector / CSR weights
  vo          the pre-multiplied V.O attention: Q|K projection, linear_vo, fused_vo_attention

Weights are N(0, 0.02^2) with small biases, activations N(0, 1), as the reference's drivers and the
tests have them; everything is fp16 with fp32 accumulation.
"""
import importlib
import math

import torch

et = importlib.import_module("scpaper-2021_b200")

# hidden width, heads, feed-forward width of the models the tests and the benchmark run
MODELS = {"d512": (512, 8, 2048), "bert-base": (768, 12, 3072), "bert-large": (1024, 16, 4096)}
MASKS = {"none": et.MASK_NONE, "causal": et.MASK_CAUSAL, "padding": et.MASK_PADDING}
VEC = 16


def _stack(name, batch, seq, model="bert-base", layers=12, mask="none", weights="dense", sparsity=0.0,
           dh_qk=64):
    return {"name": name, "kind": "stack", "model": model, "layers": layers, "batch": batch, "seq": seq,
            "mask": mask, "weights": weights, "sparsity": sparsity, "dh_qk": dh_qk}


def listed():
    return [
        # one sentence through one sparse projection: the smallest call, latency and launch
        {"name": "csr-768-t128", "kind": "csr", "tokens": 128, "in": 768, "out": 768, "sparsity": 0.95},
        # the projection of a vector-pruned model
        {"name": "1x16-1024-t3072", "kind": "1x16", "tokens": 3072, "in": 1024, "out": 3072,
         "sparsity": 0.9},
        # very sparse tiles, where the tile kernel is the recommended form
        {"name": "ffn-tile90-t2048", "kind": "ffn-tile", "tokens": 2048, "hidden": 768, "ff": 3072,
         "sparsity": 0.9},
        # pruned hidden units with full-width activations between the Linears
        {"name": "ffn-rowcol50-t3000", "kind": "ffn-rowcol", "tokens": 3000, "hidden": 768, "ff": 3072,
         "sparsity": 0.5},
        # the reference's second attention formulation at the benchmark's batch
        {"name": "vo-b16-s128", "kind": "vo", "batch": 16, "seq": 128, "hidden": 768, "heads": 12,
         "mask": "none"},
        # the reference driver's shape: one sentence, one query at a time
        _stack("stack-b1-s128", 1, 128, mask="causal"),
        # a ragged little batch of padded sentences
        _stack("stack-b5-s77", 5, 77, mask="padding"),
        # the headline configuration from and to host memory, a queue of eight batches
        {"name": "serve-b16-s128", "kind": "serve", "model": "bert-base", "layers": 12, "batch": 16,
         "seq": 128, "mask": "none", "weights": "dense", "sparsity": 0.0, "dh_qk": 64, "batches": 8},
        # 80 % tile-pruned Linears and a quarter of every head's Q/K features removed, each weight in
        # the form the plan recommends (half the depth: the layers do equal work)
        _stack("stack-b64-s128-tile80", 64, 128, layers=6, weights="tile-auto", sparsity=0.8, dh_qk=48),
        # vector-pruned projections, pruned feed-forward units, padded sequences (a quarter of the depth)
        _stack("stack-large-b32-s384-mixed", 32, 384, model="bert-large", layers=6, mask="padding",
               weights="mixed", sparsity=0.9),
        # one long document
        _stack("stack-b1-s4096", 1, 4096),
        # the scaling sweep's global batch on one GPU: the largest
        _stack("stack-b256-s512", 256, 512),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["stack"] * 6 + ["serve", "ffn-tile", "ffn-rowcol", "1x16", "csr", "vo"])
    if kind in ("stack", "serve"):
        model = rng.choice(["d512", "bert-base", "bert-base", "bert-large"])
        weights = rng.choice(["dense", "dense", "dense", "tile-auto", "tile", "mixed"])
        if kind == "serve":
            weights = "dense"
        layers = rng.randint(2, 12 if weights == "dense" else 6)
        seq = _log_int(rng, 32, 2048)
        batch = max(1, min(256, _log_int(rng, 64, 49152) // seq))
        if kind == "serve":
            batch = max(1, min(batch, 8192 // seq))
        sparsity = {"dense": 0.0, "mixed": round(rng.uniform(0.8, 0.95), 2)}.get(
            weights, round(rng.uniform(0.7, 0.95), 2))
        c = {"kind": kind, "model": model, "layers": layers, "batch": batch, "seq": seq,
             "mask": rng.choice(sorted(MASKS)), "weights": weights, "sparsity": sparsity,
             "dh_qk": 48 if weights.startswith("tile") and rng.random() < 0.5 else 64}
        if kind == "serve":
            c["batches"] = rng.randint(2, 8)
        return c
    if kind == "vo":
        seq = _log_int(rng, 32, 512)
        hidden, heads, _ = MODELS[rng.choice(sorted(MODELS))]
        return {"kind": kind, "batch": max(1, _log_int(rng, 64, 4096) // seq), "seq": seq,
                "hidden": hidden, "heads": heads, "mask": rng.choice(sorted(MASKS))}
    tokens = _log_int(rng, 64, 8192)
    hidden, _, ff = MODELS[rng.choice(sorted(MODELS))]
    if kind in ("ffn-tile", "ffn-rowcol"):
        lo, hi = (0.8, 0.95) if kind == "ffn-tile" else (0.25, 0.75)
        return {"kind": kind, "tokens": tokens, "hidden": hidden, "ff": ff,
                "sparsity": round(rng.uniform(lo, hi), 2)}
    inn, out = rng.choice([(hidden, hidden), (hidden, 3 * hidden), (hidden, ff), (ff, hidden)])
    return {"kind": kind, "tokens": tokens, "in": inn, "out": out,
            "sparsity": round(rng.uniform(0.8, 0.97), 2)}


# ---- inputs -------------------------------------------------------------------------------------

class _Gen:
    """fp16 tensors drawn on the GPU from one seed."""

    def __init__(self, seed):
        self.g = torch.Generator(device="cuda")
        self.g.manual_seed(seed)

    def normal(self, *shape, std=1.0):
        return (torch.randn(shape, generator=self.g, device="cuda") * std).half()

    def keep(self, n, sparsity):
        """Exactly floor(n * (1 - sparsity)) of n units kept, uniformly at random."""
        k = int(n * (1.0 - sparsity) + 1e-9)
        m = torch.zeros(n, dtype=torch.bool, device="cuda")
        m[torch.randperm(n, generator=self.g, device="cuda")[:k]] = True
        return m

    def ids(self, n, sparsity):
        """Sorted kept indices, a multiple of 16 of them."""
        k = max(16, int(n * (1.0 - sparsity) + 1e-9) // 16 * 16)
        return torch.randperm(n, generator=self.g, device="cuda")[:k].sort().values.int()

    def tiles(self, w, sparsity):
        out, inn = w.shape
        m = self.keep((out // 16) * (inn // 16), sparsity).view(out // 16, 1, inn // 16, 1)
        return (w.view(out // 16, 16, inn // 16, 16) * m).view(out, inn)

    def vectors(self, w, sparsity):
        out, inn = w.shape
        return (w.view(out, inn // VEC, VEC) *
                self.keep(out * (inn // VEC), sparsity).view(out, inn // VEC, 1)).view(out, inn)

    def lengths(self, batch, seq):
        lo = max(1, seq // 3)
        return torch.randint(lo, seq + 1, (batch,), generator=self.g, device="cuda", dtype=torch.int32)


def _kept_units(ff):
    return max(16, int(ff * 0.5) // 16 * 16)


def _layer(g, c):
    hidden, heads, ff = MODELS[c["model"]]
    kdim = heads * c["dh_qk"]
    w = {"wqkv": g.normal(2 * kdim + hidden, hidden, std=0.02), "bqkv": g.normal(2 * kdim + hidden, std=0.02),
         "wo": g.normal(hidden, hidden, std=0.02), "bo": g.normal(hidden, std=0.02),
         "w1": g.normal(ff, hidden, std=0.02), "b1": g.normal(ff, std=0.02),
         "w2": g.normal(hidden, ff, std=0.02), "b2": g.normal(hidden, std=0.02)}
    for ln in ("ln1", "ln2"):
        w[ln + "_g"] = g.normal(hidden, std=0.05) + 1.0
        w[ln + "_b"] = g.normal(hidden, std=0.05)
    formats, tile_sparse = None, False
    if c["weights"].startswith("tile"):
        for name in ("wqkv", "wo", "w1", "w2"):
            w[name] = g.tiles(w[name], c["sparsity"])
        tile_sparse = "auto" if c["weights"] == "tile-auto" else True
    elif c["weights"] == "mixed":
        for name in ("wqkv", "wo"):
            w[name] = g.vectors(w[name], c["sparsity"])
        ids = g.ids(ff, 0.5).cpu().numpy()
        formats = {"wqkv": "1x16_auto", "wo": "1x16_auto", "w1": ("row", ids), "w2": ("col", ids)}
    w = {k: v.cpu().numpy() for k, v in w.items()}
    return et.EncoderLayer(w, heads, et.ACT_GELU, tile_sparse=tile_sparse, formats=formats)


def prepare(case, seed):
    c, g = case, _Gen(seed)
    kind = c["kind"]
    if kind in ("stack", "serve"):
        hidden = MODELS[c["model"]][0]
        stack = et.EncoderStack([_layer(g, c) for _ in range(c["layers"])], c["batch"], c["seq"])
        s = {"kind": kind, "stack": stack, "mask": MASKS[c["mask"]],
             "valid": g.lengths(c["batch"], c["seq"]) if c["mask"] == "padding" else None}
        if kind == "stack":
            s["x"] = g.normal(c["batch"] * c["seq"], hidden)
        else:
            s["xs"] = [g.normal(c["batch"] * c["seq"], hidden).cpu().pin_memory()
                       for _ in range(c["batches"])]
            s["ys"] = [torch.empty_like(x).pin_memory() for x in s["xs"]]
            s["pipe"] = et.HostPipeline(stack, mask_kind=s["mask"], valid_len=s["valid"])
        return s
    if kind == "vo":
        hidden, heads = c["hidden"], c["heads"]
        return {"kind": kind, "case": c, "x": g.normal(c["batch"] * c["seq"], hidden),
                "wqk": g.normal(2 * hidden, hidden, std=0.02), "bqk": g.normal(2 * hidden, std=0.02),
                "wvo": g.normal(heads, hidden, hidden, std=0.01), "bo": g.normal(hidden, std=0.02),
                "valid": g.lengths(c["batch"], c["seq"]) if c["mask"] == "padding" else None}
    if kind == "ffn-tile":
        s = {"kind": kind, "x": g.normal(c["tokens"], c["hidden"])}
        for i, (out, inn) in enumerate([(c["ff"], c["hidden"]), (c["hidden"], c["ff"])], 1):
            w = g.tiles(g.normal(out, inn, std=0.02), c["sparsity"])
            s[f"w{i}"] = et.PackedTiles(*et.synth.dense_to_tile(w.cpu().numpy()), inn, out)
            s[f"b{i}"] = g.normal(out, std=0.02)
        return s
    if kind == "ffn-rowcol":
        ids = g.ids(c["ff"], c["sparsity"])
        n = int(ids.shape[0])
        return {"kind": kind, "x": g.normal(c["tokens"], c["hidden"]), "ids": ids, "ff": c["ff"],
                "rows": g.normal(n, c["hidden"], std=0.02), "cols": g.normal(c["hidden"], n, std=0.02),
                "b1": g.normal(c["ff"], std=0.02), "b2": g.normal(c["hidden"], std=0.02),
                "scratch": torch.empty((c["tokens"], n), dtype=torch.float16, device="cuda")}
    out, inn = c["out"], c["in"]
    s = {"kind": kind, "x": g.normal(c["tokens"], inn), "out": out, "bias": g.normal(out, std=0.02)}
    w = g.normal(out, inn, std=0.02)
    if kind == "csr":
        keep = g.keep(out * inn, c["sparsity"]).view(out, inn)
        s["indptr"] = torch.zeros(out + 1, dtype=torch.int32, device="cuda")
        s["indptr"][1:] = keep.sum(1).cumsum(0)
        s["indices"] = keep.nonzero()[:, 1].int().contiguous()
        s["data"] = w[keep].contiguous()
        return s
    # 1x16: vectors ordered by (set of 16 rows, part of 16 columns, row)
    nset, npart = out // 16, inn // VEC
    keep = g.keep(out * npart, c["sparsity"]).view(nset, 16, npart).transpose(1, 2)
    i = keep.nonzero()
    ends = keep.sum(2).flatten().cumsum(0).view(nset, npart)
    begin = torch.cat([ends.new_zeros(1), ends[:-1, -1]]).view(nset, 1)
    s["tile_idx"] = torch.cat([begin, ends], 1).int().flatten().contiguous()
    s["row_idx"] = (i[:, 0] * 16 + i[:, 2]).int().contiguous()
    s["data"] = w.view(nset, 16, npart, VEC)[i[:, 0], i[:, 2], i[:, 1]].contiguous()
    return s


# ---- one pass -----------------------------------------------------------------------------------

def run(state):
    s, kind = state, state["kind"]
    if kind == "stack":
        return s["stack"].forward(s["x"], s["mask"], None, s["valid"])
    if kind == "serve":
        for x, y in zip(s["xs"], s["ys"]):
            s["pipe"].submit(x, y)
        s["pipe"].drain()
        return s["ys"]
    if kind == "vo":
        c = s["case"]
        batch, seq, heads, hidden = c["batch"], c["seq"], c["heads"], c["hidden"]
        qk = et.linear_dense(s["x"], s["wqk"], s["bqk"])
        vo = et.linear_vo(s["x"], s["wvo"], None, batch, seq, heads, hidden)
        return et.fused_vo_attention(qk[:, :hidden], qk[:, hidden:], vo, s["bo"], batch, seq, heads,
                                     hidden // heads, hidden, MASKS[c["mask"]], None, s["valid"])
    if kind == "ffn-tile":
        return et.linear_tile_packed(et.linear_tile_packed(s["x"], s["w1"], s["b1"], et.ACT_GELU),
                                     s["w2"], s["b2"])
    if kind == "ffn-rowcol":
        f = et.linear_row(s["x"], s["ids"], s["rows"], s["ff"], s["b1"], et.ACT_GELU)
        return et.linear_col(f, s["ids"], s["cols"], s["b2"], scratch=s["scratch"])
    if kind == "csr":
        return et.linear_csr(s["x"], s["indptr"], s["indices"], s["data"], s["out"], s["bias"])
    return et.linear_1x16(s["x"], s["tile_idx"], s["row_idx"], s["data"], s["out"], s["bias"])


# ---- what a pass cannot do without --------------------------------------------------------------

def _pairs(seq, mask):
    """(query, key) pairs of one sequence; padded lengths average two thirds of seq."""
    return {"none": seq * seq, "causal": seq * (seq + 1) / 2, "padding": seq * seq * 2 / 3}[mask]


def work(case):
    c, kind = case, case["kind"]
    if kind in ("stack", "serve"):
        hidden, heads, ff = MODELS[c["model"]]
        T, kdim = c["batch"] * c["seq"], heads * c["dh_qk"]
        proj, ffn = (2 * kdim + 2 * hidden) * hidden, 2 * hidden * ff
        index = 0.0
        if c["weights"].startswith("tile"):
            stored = (proj + ffn) * (1 - c["sparsity"])
            index = stored / 256 * 4
        elif c["weights"] == "mixed":
            kept = proj * (1 - c["sparsity"])
            stored = kept + 2 * hidden * _kept_units(ff)
            index = kept / VEC * 4
        else:
            stored = proj + ffn
        n = c.get("batches", 1)
        attn = 2 * c["batch"] * _pairs(c["seq"], c["mask"]) * (kdim + hidden)
        return {"bytes": c["layers"] * (2 * stored + index) + n * 2 * T * hidden * 2,
                "flops": n * c["layers"] * (2 * T * stored + attn)}
    if kind == "vo":
        h, T = c["hidden"], c["batch"] * c["seq"]
        pairs = c["batch"] * _pairs(c["seq"], c["mask"])
        return {"bytes": 2 * (2 * T * h + 2 * h * h + c["heads"] * h * h),
                "flops": 2 * T * h * h * (2 + c["heads"]) + 2 * pairs * h * (1 + c["heads"])}
    T = c["tokens"]
    if kind == "ffn-tile":
        stored = 2 * c["hidden"] * c["ff"] * (1 - c["sparsity"])
        return {"bytes": 2 * stored * (1 + 2 / 256) + 4 * T * c["hidden"], "flops": 2 * T * stored}
    if kind == "ffn-rowcol":
        stored = 2 * c["hidden"] * max(16, int(c["ff"] * (1 - c["sparsity"])) // 16 * 16)
        return {"bytes": 2 * stored + 4 * T * c["hidden"], "flops": 2 * T * stored}
    stored = c["in"] * c["out"] * (1 - c["sparsity"])
    index = 4 * stored if kind == "csr" else 4 * stored / VEC
    return {"bytes": 2 * stored + index + 2 * T * (c["in"] + c["out"]), "flops": 2 * T * stored}


def tolerance(case):
    # fp16 storage of every tensor between operators, fp32 accumulation: a single Linear differs by
    # the rounding of its output, a stack by what up to twelve layers make of such roundings
    if case["kind"] in ("stack", "serve"):
        return {"rel": 3e-3, "max": 3e-2}
    if case["kind"] in ("csr", "1x16"):
        return {"rel": 5e-4, "max": 5e-3}
    return {"rel": 1.5e-3, "max": 1.5e-2}
