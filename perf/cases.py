"""The work that users of this package have it do, as cases that can be timed.

Six paths, all through public entry points:

* ``linear``   one :class:`LutLinear` forward: row-wise scales or the block ("Lat.") layouts, from one decoded token to
               the rows of a prompt;
* ``set``      the linear layers of decoder blocks as prepared grouped launches, chained with programmatic dependent launch;
* ``decode``   one token of :class:`BcqLlamaDecoder` (the captured CUDA graph), fp16 or fixed-point accumulator outputs;
* ``batch``    one step of :class:`BcqLlamaBatchDecoder`: sequences in lock step;
* ``prefill``  a prompt through :meth:`BcqLlamaDecoder.prefill`;
* ``convert``  a "Lat." checkpoint tensor brought into the kernels' layout when a model is loaded.

Weights are synthetic: packed sign bits i.i.d. uniform, activations N(0, 1) in fp16.  ``scales``: "pow2" = 2**-k with
k uniform in 2..8 (the power-of-two recipe of the synthetic layers), "real" = the same exponents with a uniform
mantissa (scales that were fitted and not rounded to powers of two).
"""
import math

import torch

from shiftaddllm_b200 import lutgemm
from shiftaddllm_b200.decoder import BcqLlamaBatchDecoder, BcqLlamaDecoder, LlamaShape
from shiftaddllm_b200.kernel import convert_weight
from shiftaddllm_b200.quant import LutLinear

# LLaMA-2-7B and 70B decoder dimensions (the configurations of the benchmark and of decoder.SHAPES)
_7B = {"hidden": 4096, "heads": 32, "kv_heads": 32, "ffn": 11008, "vocab": 32000}


def listed():
    return [
        # the smallest layer of the test configurations (OPT-125m q_proj, with bias), one token: launches and host work count
        {"name": "linear_768_token", "path": "linear", "layout": "row", "K": 768, "N": 768, "q": 3, "g": 128, "rows": 1, "bias": True, "scales": "pow2"},
        # a 7B attention projection in the layout LutLinear.forward of the reference calls (int8 exponent triples), one token
        {"name": "linear_lat_i8_token", "path": "linear", "layout": "block_i8", "K": 4096, "N": 4096, "q": 3, "g": 16, "rows": 1, "bias": False, "scales": "pow2"},
        # the same family of layers as the checkpoint loader leaves them by default (fp16 multipliers), the rows of a prompt
        {"name": "linear_lat_f16_prompt", "path": "linear", "layout": "block_f16", "K": 11008, "N": 4096, "q": 3, "g": 16, "rows": 128, "bias": False, "scales": "real"},
        # a 4-bit 7B gate projection for eight sequences
        {"name": "linear_gate_rows8", "path": "linear", "layout": "row", "K": 4096, "N": 11008, "q": 4, "g": 128, "rows": 8, "bias": False, "scales": "real"},
        # sizes that are no multiple of anything large, small groups, bias, a few rows
        {"name": "linear_ragged", "path": "linear", "layout": "row", "K": 2080, "N": 1378, "q": 3, "g": 32, "rows": 3, "bias": True, "scales": "real"},
        # the largest single layer: 70B down projection, 2 bit, one token
        {"name": "linear_70b_down_token", "path": "linear", "layout": "row", "K": 28672, "N": 8192, "q": 2, "g": 128, "rows": 1, "bias": False, "scales": "pow2"},
        # the seven linears of 7B decoder blocks as one grouped launch per block (what the benchmark's headline times)
        {"name": "set_7b", "path": "set", "layers": 4, "hidden": 4096, "kv": 4096, "ffn": 11008, "q": 3, "g": 128, "rows": 1, "ordered": False},
        # one decoded token of the 7B decoder at position 512, fp16 outputs (the default) and fixed-point accumulators
        {"name": "decode_7b", "path": "decode", "layers": 32, **_7B, "q": 3, "g": 128, "pos": 512, "atomic": False},
        {"name": "decode_7b_fixed", "path": "decode", "layers": 32, **_7B, "q": 3, "g": 128, "pos": 512, "atomic": True},
        # sixteen sequences in lock step
        {"name": "batch16_7b", "path": "batch", "layers": 32, **_7B, "q": 3, "g": 128, "pos": 512, "batch": 16},
        # a 512-token prompt
        {"name": "prefill_7b", "path": "prefill", "layers": 32, **_7B, "q": 3, "g": 128, "tokens": 512},
        # loading: one 7B down projection from the checkpoint's packing into the kernels'
        {"name": "convert_7b_down", "path": "convert", "K": 11008, "N": 4096, "q": 3, "g": 16},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    path = rng.choice(["linear"] * 6 + ["set", "decode", "decode", "batch", "prefill", "convert"])
    q = rng.choice((2, 3, 3, 4))
    if path == "linear":
        layout = rng.choice(("row", "row", "block_f16", "block_i8"))
        rows = rng.choice((1, 1, _log(rng, 1, 64), _log(rng, 1, 256)))
        scales = "pow2" if layout == "block_i8" else rng.choice(("pow2", "real"))
        case = {"path": path, "layout": layout, "q": q, "rows": rows, "bias": rng.random() < 0.4, "scales": scales}
        if rng.random() < 0.25:   # ragged: K a multiple of 32 only, N of what its groups ask for
            g = 32 if layout == "row" else 16
            k, n = 32 * _log(rng, 8, 160), 2 * _log(rng, 64, 2048)
            return {**case, "K": k, "N": n if layout == "row" else max(16, n // 16 * 16), "g": g}
        k, n = 256 * _log(rng, 2, 112), 64 * _log(rng, 4, 448)
        while k * n > 28672 * 8192:
            k, n = max(256, k // 2 // 256 * 256), max(64, n // 2 // 64 * 64)
        return {**case, "K": k, "N": n, "g": rng.choice((128, 128, 256)) if layout == "row" else 16}
    if path == "convert":
        return {"path": path, "K": 32 * _log(rng, 16, 896), "N": 128 * _log(rng, 4, 64), "q": q, "g": 16}
    heads = rng.choice((8, 16, 24, 32, 32, 40, 64))
    hidden, kv_heads = 128 * heads, rng.choice((heads, heads, 8))
    ffn, layers = 256 * rng.randint(hidden // 128, 7 * hidden // 512), rng.randint(1, 8 if hidden > 4096 else 16)
    if path == "set":
        return {"path": path, "layers": min(layers, 9), "hidden": hidden, "kv": 128 * kv_heads, "ffn": ffn, "q": q, "g": 128,
                "rows": rng.choice((1, 1, _log(rng, 1, 64))), "ordered": rng.random() < 0.5}
    case = {"path": path, "layers": layers, "hidden": hidden, "heads": heads, "kv_heads": kv_heads, "ffn": ffn, "vocab": 32000, "q": q, "g": 128}
    if path == "decode":
        return {**case, "pos": _log(rng, 8, 1000), "atomic": rng.random() < 0.5}
    if path == "batch":
        return {**case, "pos": _log(rng, 8, 600), "batch": _log(rng, 2, 48)}
    return {**case, "tokens": _log(rng, 16, 512)}


# ---- what a program has in hand before the call ---------------------------------------------------------------------
def _bits(gen, *shape):
    return torch.randint(-2 ** 31, 2 ** 31, shape, dtype=torch.int32, device="cuda", generator=gen)


def _scales(gen, kind, *shape):
    a = torch.exp2(-torch.randint(2, 9, shape, device="cuda", generator=gen).float())
    return a if kind == "pow2" else a * (0.5 + 0.5 * torch.rand(shape, device="cuda", generator=gen))


def _linear(case, gen):
    k, n, q, g = case["K"], case["N"], case["q"], case["g"]
    row = case["layout"] == "row"
    lin = LutLinear(k, n, g if row else 8 * g, q)
    lin.binaryWeight = _bits(gen, k // 32, q, n)
    if row:
        lin.set_row_alpha(_scales(gen, case["scales"], k // g, q, n))
    else:
        lin.set_block_alpha(_scales(gen, case["scales"], k // 8, q, n // g), apot=case["layout"] == "block_i8")
    if case["bias"]:
        lin.bias = (0.02 * torch.randn(n, device="cuda", generator=gen)).half()
    return {"layer": lin, "x": torch.randn(case["rows"], k, device="cuda", generator=gen).half()}


def _set(case, gen):
    h, kv, ffn, q, g, m = (case[f] for f in ("hidden", "kv", "ffn", "q", "g", "rows"))
    launches, outputs = [], []
    for _ in range(case["layers"]):
        block = []
        for k, n in ((h, h), (h, kv), (h, kv), (h, h), (h, ffn), (h, ffn), (ffn, h)):
            y = torch.empty(m, n, dtype=torch.float16, device="cuda")
            outputs.append(y)
            block.append(dict(output=y, bWeight=_bits(gen, k // 32, q, n), alpha=_scales(gen, "pow2", k // g, q, n).half(), bias=None,
                              d_input=torch.randn(m, k, device="cuda", generator=gen).half(), mSize=n, kSize=k, nb=q, num_groups=k // g))
        groups = ((0, 3), (3, 4), (4, 6), (6, 7)) if case["ordered"] else ((0, 7),)   # in the order of a decoder's dependencies, or all at once
        launches += [lutgemm.prepare_grouped(block[a:b], pdl=True) for a, b in groups]
    return {"sequence": lutgemm.LaunchSequence(launches), "outputs": outputs}


def _shape(case):
    return LlamaShape(case["hidden"], case["layers"], case["heads"], case["kv_heads"], case["ffn"], vocab=case["vocab"])


def _model(case, gen, seed, cls, max_len, **more):
    """A decoder with seeded weights.  The synthetic scales (2**-2 .. 2**-8) are brought to those of trained weights
    (standard deviation of a weight about 0.006), so that activations stay of order one over the layers."""
    model = cls(_shape(case), case["q"], case["g"], max_len=max_len, seed=seed, **more)
    for block in model.blocks:
        for lin in block.linears().values():
            lin.alpha.mul_(2.0 ** -5)
    return model


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    path = case["path"]
    with torch.no_grad():
        if path == "linear":
            state = _linear(case, gen)
        elif path == "set":
            state = _set(case, gen)
        elif path == "convert":
            k, n, q, g = (case[f] for f in "KNqg")
            state = {"planes": _bits(gen, k, n // 32, q), "alpha": _scales(gen, "real", k // 8, n // g, q)}
        elif path == "prefill":
            model = _model(case, gen, seed, BcqLlamaDecoder, case["tokens"] + 64)
            state = {"model": model, "ids": torch.randint(0, case["vocab"], (case["tokens"],), device="cuda", generator=gen)}
        else:
            if path == "decode":
                model = _model(case, gen, seed, BcqLlamaDecoder, case["pos"] + 128, atomic=case["atomic"])
            else:
                model = _model(case, gen, seed, BcqLlamaBatchDecoder, case["pos"] + 128, batch=case["batch"])
            # keys and values of the positions decoded so far; the later ones are zero until they are written
            seen = (slice(None),) * (1 if path == "decode" else 2) + (slice(0, case["pos"]),)
            for cache in (model.k_cache, model.v_cache):
                cache[seen] = torch.randn(cache[seen].shape, dtype=torch.float16, device="cuda", generator=gen)
            torch.cuda.synchronize()   # capture() takes its warm-up step on a stream of its own
            model.capture()
            state = {"model": model, "pos": torch.full_like(model.pos, case["pos"]),
                     "token": torch.randint(0, case["vocab"], model.token.shape, device="cuda", generator=gen)}
    state["path"] = path
    return state


# ---- one pass ---------------------------------------------------------------------------------------------------------
def run(state):
    path = state["path"]
    with torch.no_grad():
        if path == "linear":
            return state["layer"](state["x"])
        if path == "set":
            state["sequence"]()
            return state["outputs"]
        if path == "convert":
            return convert_weight(state["planes"], state["alpha"])
        model = state["model"]
        if path == "prefill":
            model.pos.zero_()
            model.prefill(state["ids"])
        else:
            model.token.copy_(state["token"])   # the token and the position that a serving loop hands in
            model.pos.copy_(state["pos"])
            model.graph.replay()
        return {"logits": model.logits, "keys": model.k_cache, "values": model.v_cache}


# ---- what a pass cannot do without ------------------------------------------------------------------------------------
def _product(rows, k, n, q, scale_bytes, bias=False):
    return {"bytes": k * n * q // 8 + scale_bytes + (2 * n if bias else 0) + 2 * rows * (k + n), "flops": 2 * rows * k * n}


def work(case):
    path, q = case["path"], case["q"]
    if path == "convert":
        k, n, g = case["K"], case["N"], case["g"]
        scales = (k // 8) * (n // g) * q
        return {"bytes": 2 * (k * n * q // 8) + 2 * 4 * scales, "flops": 0}
    if path == "linear":
        k, n, g = case["K"], case["N"], case["g"]
        scales = {"row": 2 * (k // g) * n, "block_f16": 2 * (k // 8) * (n // g), "block_i8": 3 * (k // 8) * (n // g)}[case["layout"]] * q
        return _product(case["rows"], k, n, q, scales, case["bias"])
    h, ffn, g = case["hidden"], case["ffn"], case["g"]
    kv = case["kv"] if path == "set" else 128 * case["kv_heads"]
    rows = {"set": case.get("rows"), "decode": 1, "batch": case.get("batch"), "prefill": case.get("tokens")}[path]
    total = {"bytes": 0, "flops": 0}
    for k, n in ((h, h), (h, kv), (h, kv), (h, h), (h, ffn), (h, ffn), (ffn, h)):
        w = _product(rows, k, n, q, 2 * (k // g) * n * q)
        for f in total:
            total[f] += case["layers"] * w[f]
    if path == "set":
        return total
    # keys and values: read up to the position, written at it; attention; the output head in fp16
    last = case["tokens"] if path == "prefill" else case["pos"]
    total["bytes"] += case["layers"] * 2 * 2 * kv * (rows if path != "decode" else 1) * (1 if path == "prefill" else last + 1)
    total["flops"] += case["layers"] * 4 * h * (last * (last + 1) // 2 if path == "prefill" else rows * (last + 1))
    heads_out = 1 if path == "prefill" else rows
    total["bytes"] += 2 * h * case["vocab"] + 2 * rows * h + 4 * heads_out * case["vocab"]
    total["flops"] += 2 * heads_out * h * case["vocab"]
    return total


def tolerance(case):
    """About four times what each path shows against the same computation in float64: the rounding of the fp16 output
    (2.1e-4, largest 4.9e-4), of fp16 table entries in the row-scaled small-batch product (4.4e-4, largest 2.2e-3), and of
    fp16 activations and outputs over the layers of a decoder (3.5e-3 for a token, 4.5e-3 for a batch, 1.7e-3 for a prompt)."""
    path = case["path"]
    if path == "convert":
        return "exact"
    if path in ("linear", "set"):
        small_batch = case["rows"] > 1 and case.get("layout", "row") == "row"
        return {"rel": 1.7e-3, "max": 9e-3} if small_batch else {"rel": 8.5e-4, "max": 2e-3}
    return {"decode": {"rel": 1.4e-2, "max": 6.5e-2}, "batch": {"rel": 1.8e-2, "max": 9e-2}, "prefill": {"rel": 7e-3, "max": 4e-2}}[path]


# ---- the same in 64 bits, in plain torch ------------------------------------------------------------------------------
def _dense(packed, scales):
    """Packed planes [K/32, q, N] and scales [., q, .] (rows of the scales: equal runs of K, columns: equal runs of N) as a float64 weight [K, N]."""
    words, q, n = packed.shape
    k = 32 * words
    shifts = torch.arange(32, device=packed.device, dtype=torch.int32).view(1, 32, 1)
    weight = torch.zeros(k, n, dtype=torch.float64, device=packed.device)
    for b in range(q):
        a = scales[:, b].double().repeat_interleave(n // scales.shape[2], dim=1)   # [runs of K, N]
        for lo in range(0, words, 128):
            sign = ((packed[lo:lo + 128, b][:, None, :] >> shifts) & 1).reshape(-1, n).double().mul_(2).sub_(1)
            rows = torch.arange(32 * lo, 32 * lo + sign.shape[0], device=packed.device) // (k // scales.shape[0])
            weight[32 * lo:32 * lo + sign.shape[0]] += sign.mul_(a[rows])
    return weight


def _layer(lin, x):
    a = lin.alpha
    if a.dtype == torch.int8:   # three exponents a multiplier, -128 for one that is not there
        a = torch.where(a == -128, torch.zeros((), dtype=torch.float64, device=a.device), torch.exp2(a.double())).sum(-1)
    y = x @ _dense(lin.binaryWeight, a)
    return y if lin.bias is None else y + lin.bias.double()


def _norm(x, w, eps):
    return x * torch.rsqrt((x * x).mean(-1, keepdim=True) + eps) * w.double()


def _tokens(model, shape, ids, keys, values, first):
    """`ids` [sequences, tokens] at positions first, first + 1, ..: the logits of the last token of each sequence; their keys
    and values are written into `keys`, `values` [layers, sequences, positions, kv heads, head dim]."""
    hd, kvh, rep = shape.head_dim, shape.kv_heads, shape.heads // shape.kv_heads
    s, t = ids.shape
    dev = ids.device
    at = torch.arange(first, first + t, device=dev)
    angle = at.double()[:, None] / shape.rope_theta ** (torch.arange(0, hd, 2, device=dev).double() / hd)
    cos, sin = angle.cos()[None, :, None], angle.sin()[None, :, None]

    def turned(v, heads):
        a, b = v.view(s, t, heads, 2, hd // 2).unbind(3)
        return torch.cat((a * cos - b * sin, b * cos + a * sin), dim=-1)

    later = torch.arange(first + t, device=dev)[None, :] > at[:, None]
    x = model.embed[ids].double()
    for i, blk in enumerate(model.blocks):
        h = _norm(x, blk.input_norm, shape.eps)
        qh = turned(_layer(blk.q_proj, h), shape.heads)
        keys[i, :, first:first + t] = turned(_layer(blk.k_proj, h), kvh)
        values[i, :, first:first + t] = _layer(blk.v_proj, h).view(s, t, kvh, hd)
        k, v = (c[i, :, :first + t].double().repeat_interleave(rep, dim=2) for c in (keys, values))
        scores = torch.einsum("sthd,sphd->shtp", qh, k) / math.sqrt(hd)
        p = torch.softmax(scores.masked_fill(later, float("-inf")), dim=-1)
        x = x + _layer(blk.o_proj, torch.einsum("shtp,sphd->sthd", p, v).reshape(s, t, -1))
        h = _norm(x, blk.post_norm, shape.eps)
        x = x + _layer(blk.down_proj, torch.nn.functional.silu(_layer(blk.gate_proj, h)) * _layer(blk.up_proj, h))
    return _norm(x[:, -1], model.final_norm, shape.eps) @ model.lm_head.double().t()


def exact(case, seed):
    path, state = case["path"], prepare(case, seed)
    with torch.no_grad():
        if path == "linear":
            return _layer(state["layer"], state["x"].double())
        if path == "set":
            out = []
            for launch in state["sequence"]._launches:
                for _, bits, scales, _, x, _ in launch._keep:
                    out.append(x.double() @ _dense(bits, scales))
            return out
        if path == "convert":
            return None, state["alpha"].double().transpose(1, 2)
        model, shape = state["model"], _shape(case)
        keys, values = model.k_cache.float(), model.v_cache.float()   # given ones are fp16 numbers; those computed here are rounded to 32 bits
        if path == "batch":
            logits = _tokens(model, shape, state["token"].view(-1, 1), keys, values, case["pos"])
        else:
            ids, first = (state["ids"], 0) if path == "prefill" else (state["token"], case["pos"])
            logits = _tokens(model, shape, ids.view(1, -1), keys[:, None], values[:, None], first)[0]
        return {"logits": logits, "keys": keys, "values": values}
