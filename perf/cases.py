"""The work that programs built on this framework have it do, as cases that can be timed and compared.

Seven kinds of case, each through entry points of the C ABI (include/b200_ggml.h, include/b200_ggml_ops.h) or of the decoder:

  proj    the attention projections of a quantised decoder layer: RMS norm, q / k / v, output product (+ residual when decoding)
  mlp     its gated feed-forward: RMS norm, gate / up, SiLU, down (+ residual when decoding)
  moe     its routed feed-forward: expert gate / up, SiLU, expert down for given expert ids
  attn    FLASH_ATTN_EXT over an f16 or q8_0 cache, decoding or a prompt batch with a causal mask
  block   the attention of a layer served from a folder in bf16: q | k | v product, rotation + cache store, attention with a sink, output product
  delta   a recurrent mixer of such a layer: short convolution, then the gated delta rule
  model   whole calls of the decoder: single tokens, host tokens in, host logits out

Sizes are those of the model shapes that the framework names (TinyLlama, Llama-2 7B / 13B, Mixtral 8x7B, the design benchmarks at width
4096) and, for drawn cases, spread between them.
"""
import ctypes as C
import math

import numpy as np
import torch

from koboldcpp_b200 import llama
from koboldcpp_b200.lib import (BF16, F16, F32, Q4_0, Q4_K, Q5_K, Q6_K, Q8_0, DeltaRuleArgs, FattnArgs, GemvFuse, GemvJob, QkvStoreArgs, ShortConvArgs,
                                SinkAttnArgs, Tensor, check, lib)

TYPES = {"q4_0": Q4_0, "q8_0": Q8_0, "q4_K": Q4_K, "q5_K": Q5_K, "q6_K": Q6_K, "f16": F16, "bf16": BF16}
BLOCK = {"q4_0": (32, 18), "q8_0": (32, 34), "q4_K": (256, 144), "q5_K": (256, 176), "q6_K": (256, 210)}  # values, bytes
EPS = 1e-5


def row_bytes(kind, k):
    values, size = BLOCK[kind]
    return k // values * size


# ------------------------------------------------------------------------------------------------ inputs
def generator(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def normal(g, *shape, std=1.0):
    return torch.randn(*shape, generator=g, device="cuda") * std


def activations(g, tokens, width):
    """Rows of a residual stream: normal values, one channel in a hundred much louder, as trained models have them."""
    loud = 1.0 + 7.0 * (torch.rand(width, generator=g, device="cuda") < 0.01)
    return normal(g, tokens, width) * loud


def quantised(g, kind, rows, k, gain=1.0):
    """Random blocks: uniform quants and sub-block scales under super-block scales that give weights of mean 0 and deviation about 0.02 * gain."""
    values, size = BLOCK[kind]
    n = k // values
    raw = torch.randint(0, 256, (rows, n, size), generator=g, device="cuda", dtype=torch.uint8)

    def put(at, lo, hi, *more):
        d = (torch.rand(rows, n, generator=g, device="cuda") * (hi - lo) + lo) * gain
        for i, factor in enumerate((1.0,) + more):
            raw[:, :, at + 2 * i:at + 2 * i + 2] = (d * factor).half().view(torch.uint8).reshape(rows, n, 2)

    if kind == "q4_0":
        put(0, 3e-3, 5.5e-3)
        q = raw[:, :, 2:]  # quants -8 to 7: those at -8, which would pull the mean off 0, become 0
        q += 8 * (q & 15 == 0).byte() + 128 * (q >> 4 == 0).byte()
    elif kind == "q8_0":
        put(0, 2e-4, 3.4e-4)
    elif kind in ("q4_K", "q5_K"):
        put(0, *((1.1e-4, 1.9e-4, 7.5) if kind == "q4_K" else (4.5e-5, 7.5e-5, 15.5)))
        # a sub-block's minimum has the bits of its scale, so that its values lie around 0
        raw[:, :, 8:12] = raw[:, :, 4:8]
        raw[:, :, 12:16] = (raw[:, :, 12:16] & 15) * 17
    else:
        put(208, 1.1e-5, 1.9e-5)
    # one flat allocation with room behind the last row: kernels may read up to the next 16-byte boundary
    flat = torch.zeros(raw.numel() + 256, dtype=torch.uint8, device="cuda")
    flat[:raw.numel()] = raw.reshape(-1)
    return flat


def dequantised(flat, kind, rows, k):
    """The blocks' values in 64 bits, by the definition of the format."""
    values, size = BLOCK[kind]
    n = k // values
    b = flat[:rows * n * size].reshape(rows, n, size)

    def half(at):
        return b[:, :, at:at + 2].contiguous().view(torch.float16).double()

    if kind == "q4_0":
        q = b[:, :, 2:].short()
        return (half(0) * torch.cat([(q & 15) - 8, (q >> 4) - 8], dim=2)).reshape(rows, k)
    if kind == "q8_0":
        return (half(0) * b[:, :, 2:].contiguous().view(torch.int8).double()).reshape(rows, k)
    if kind in ("q4_K", "q5_K"):
        s = b[:, :, 4:16].short()
        scale = torch.cat([s[:, :, :4] & 63, (s[:, :, 8:] & 15) | ((s[:, :, :4] >> 6) << 4)], dim=2)
        low = torch.cat([s[:, :, 4:8] & 63, (s[:, :, 8:] >> 4) | ((s[:, :, 4:8] >> 6) << 4)], dim=2)
        q = b[:, :, size - 128:].short().reshape(rows, n, 4, 1, 32)
        q = torch.cat([q & 15, q >> 4], dim=3).reshape(rows, n, 8, 32)
        if kind == "q5_K":
            bit = torch.arange(8, device="cuda", dtype=torch.int16).reshape(1, 1, 8, 1)
            q = q + (((b[:, :, 16:48].short().reshape(rows, n, 1, 32) >> bit) & 1) << 4)
        return (half(0).unsqueeze(3) * scale.unsqueeze(3) * q - half(2).unsqueeze(3) * low.unsqueeze(3)).reshape(rows, k)
    ql, qh = b[:, :, :128].short().reshape(rows, n, 2, 2, 32), b[:, :, 128:192].short().reshape(rows, n, 2, 1, 32)
    scale = b[:, :, 192:208].contiguous().view(torch.int8).double().reshape(rows, n, 2, 4, 2, 1)
    quarter = torch.arange(4, device="cuda", dtype=torch.int16).reshape(1, 1, 1, 4, 1)
    q = torch.cat([ql & 15, ql >> 4], dim=3) | (((qh >> (2 * quarter)) & 3) << 4)
    return (half(208).reshape(rows, n, 1, 1, 1, 1) * scale * (q - 32).reshape(rows, n, 2, 4, 2, 16)).reshape(rows, k)


def tensor(t, *ne, kind=F32):
    return Tensor.contiguous(t.data_ptr(), kind, ne)


def product(kind, w, x, dst, rows, k, tokens, ws, again=False):
    """A prompt's product; `again`: the activations of the call before, which the workspace still holds."""
    check(lib().b200_mul_mat_q(TYPES[kind], w.data_ptr(), 2 * k if kind == "bf16" else row_bytes(kind, k), None if again else x.data_ptr(), k, dst.data_ptr(), rows, k, rows,
                               tokens, ws.data_ptr(), ws.numel(), None), "b200_mul_mat_q")


def vector(kind, w, x, dst, rows, k, tokens):
    check(lib().b200_mul_mat_vec_q(TYPES[kind], w.data_ptr(), row_bytes(kind, k), x.data_ptr(), k, dst.data_ptr(), rows, k, rows, tokens, None), "b200_mul_mat_vec_q")


def workspace(nbytes):
    return torch.zeros(int(nbytes) + 256, dtype=torch.uint8, device="cuda")


def product_ws(kind, k, rows, tokens):
    return workspace(lib().b200_mul_mat_q_workspace_bytes(TYPES[kind], k, rows, tokens))


def fused(jobs, norm=None, residual=None, silu=False):
    """Arguments of a decoding launch: (weight, input, output, rows) per job."""
    a = (GemvJob * len(jobs))()
    for i, (w, x, dst, rows) in enumerate(jobs):
        a[i].W, a[i].X, a[i].dst, a[i].M, a[i].id_index = w.data_ptr(), x.data_ptr(), dst, rows, -1
    f = GemvFuse()
    if norm is not None:
        f.norm_weight, f.norm_eps = norm.data_ptr(), EPS
    if residual is not None:
        f.residual[0] = residual.data_ptr()
    f.silu_pair = 1 if silu else 0
    return a, len(jobs), f


def launch(kind, args, k, out_stride, tokens):
    check(lib().b200_mul_mat_vec_q_fused(TYPES[kind], args[0], args[1], row_bytes(kind, k), k, out_stride, k, tokens, C.byref(args[2]), None), "b200_mul_mat_vec_q_fused")


def rms64(x, w=None):
    y = x.double() / torch.sqrt(x.double().square().mean(-1, keepdim=True) + EPS)
    return y if w is None else y * w.double()


def silu64(x):
    return x * torch.sigmoid(x)


def spread(rng, lo, hi):
    """A whole number, spread over its logarithm."""
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def tokens_of(rng):
    """Half the calls decode (1 to 8 tokens at once), half bring a prompt."""
    return rng.choice([1, 1, 2, 3, 4, 5, 7, 8]) if rng.random() < 0.5 else spread(rng, 9, 512)


class Proj:
    """q, k and v of one layer read the same normalised rows; the output product reads the attention's result."""

    @staticmethod
    def draw(rng):
        dim, group = rng.choice([64, 128]), rng.choice([1, 4, 8])
        kv_heads = max(1, spread(rng, 8, 40) // group)
        width = -(-kv_heads * group * dim // 256) * 256
        kind = rng.choice(["q4_0", "q8_0", "q4_K", "q5_K", "q6_K"])
        return {"width": width, "kv_width": kv_heads * dim, "type": kind, "type_v": "q6_K" if kind in ("q4_K", "q5_K") and rng.random() < 0.5 else kind, "tokens": tokens_of(rng)}

    @staticmethod
    def weights(c, g):
        n, kv = c["width"], c["kv_width"]
        return {"norm": 1 + normal(g, n, std=0.1), "q": quantised(g, c["type"], n, n), "k": quantised(g, c["type"], kv, n), "v": quantised(g, c["type_v"], kv, n),
                "o": quantised(g, c["type"], n, n), "x": activations(g, c["tokens"], n), "mix": normal(g, c["tokens"], n, std=0.5)}

    @staticmethod
    def prepare(c, seed):
        s = Proj.weights(c, generator(seed))
        n, kv, t = c["width"], c["kv_width"], c["tokens"]
        s["h"] = torch.empty(t, n, device="cuda")
        if t <= 4:
            # one row of the result holds q | k | v: the products of a launch share a row stride
            same = c["type"] == c["type_v"]
            s["qkv"] = torch.empty(t, n + 2 * kv, device="cuda")
            at = s["qkv"].data_ptr()
            s["first"] = fused([(s["q"], s["x"], at, n), (s["k"], s["x"], at + 4 * n, kv)] + ([(s["v"], s["x"], at + 4 * (n + kv), kv)] if same else []), norm=s["norm"])
            s["second"] = None if same else fused([(s["v"], s["x"], at + 4 * (n + kv), kv)], norm=s["norm"])
            s["out"] = torch.empty(t, n, device="cuda")
            s["last"] = fused([(s["o"], s["mix"], s["out"].data_ptr(), n)], residual=s["x"])
        else:
            s["qo"], s["ko"], s["vo"], s["out"] = (torch.empty(t, m, device="cuda") for m in (n, kv, kv, n))
            s["ws"] = product_ws(c["type"], n, n, t) if t > 8 else None
        return s

    @staticmethod
    def run(c, s):
        n, kv, t = c["width"], c["kv_width"], c["tokens"]
        if t <= 4:
            launch(c["type"], s["first"], n, n + 2 * kv, t)
            if s["second"]:
                launch(c["type_v"], s["second"], n, n + 2 * kv, t)
            launch(c["type"], s["last"], n, n, t)
            return [s["qkv"], s["out"]]
        check(lib().b200_op_rms_norm_mul(C.byref(tensor(s["x"], n, t)), s["norm"].data_ptr(), None, C.byref(tensor(s["h"], n, t)), EPS, None))
        if t <= 8:
            vector(c["type"], s["q"], s["h"], s["qo"], n, n, t)
            vector(c["type"], s["k"], s["h"], s["ko"], kv, n, t)
            vector(c["type_v"], s["v"], s["h"], s["vo"], kv, n, t)
            vector(c["type"], s["o"], s["mix"], s["out"], n, n, t)
        else:
            product(c["type"], s["q"], s["h"], s["qo"], n, n, t, s["ws"])
            product(c["type"], s["k"], s["h"], s["ko"], kv, n, t, s["ws"], again=True)
            product(c["type_v"], s["v"], s["h"], s["vo"], kv, n, t, s["ws"], again=True)
            product(c["type"], s["o"], s["mix"], s["out"], n, n, t, s["ws"])
        return [s["qo"], s["ko"], s["vo"], s["out"]]

    @staticmethod
    def exact(c, seed):
        s = Proj.weights(c, generator(seed))
        n, kv, t = c["width"], c["kv_width"], c["tokens"]
        h = rms64(s["x"], s["norm"])
        q, k = h @ dequantised(s["q"], c["type"], n, n).T, h @ dequantised(s["k"], c["type"], kv, n).T
        v, o = h @ dequantised(s["v"], c["type_v"], kv, n).T, s["mix"].double() @ dequantised(s["o"], c["type"], n, n).T
        return [torch.cat([q, k, v], dim=1), o + s["x"]] if t <= 4 else [q, k, v, o]

    @staticmethod
    def work(c):
        n, kv, t = c["width"], c["kv_width"], c["tokens"]
        weights = row_bytes(c["type"], n) * (2 * n + kv) + row_bytes(c["type_v"], n) * kv
        return {"bytes": weights + 4 * t * (4 * n + 2 * kv), "flops": 2 * t * n * (2 * n + 2 * kv)}


class Mlp:
    @staticmethod
    def draw(rng):
        return {"width": 256 * spread(rng, 4, 20), "ff": 256 * spread(rng, 8, 54), "type": rng.choice(["q4_0", "q8_0", "q4_K", "q5_K", "q6_K"]),
                "type_down": rng.choice(["q4_K", "q6_K", "q5_K", "q4_0"]), "tokens": tokens_of(rng)}

    @staticmethod
    def weights(c, g):
        n, ff = c["width"], c["ff"]
        return {"norm": 1 + normal(g, n, std=0.1), "gate": quantised(g, c["type"], ff, n), "up": quantised(g, c["type"], ff, n), "down": quantised(g, c["type_down"], n, ff),
                "x": activations(g, c["tokens"], n)}

    @staticmethod
    def prepare(c, seed):
        s = Mlp.weights(c, generator(seed))
        n, ff, t = c["width"], c["ff"], c["tokens"]
        s["h"], s["out"] = torch.empty(t, n, device="cuda"), torch.empty(t, n, device="cuda")
        s["g"], s["u"], s["act"] = (torch.empty(t, ff, device="cuda") for _ in range(3))
        if t <= 4:
            first = s["act"] if t == 1 else s["g"]
            s["first"] = fused([(s["gate"], s["x"], first.data_ptr(), ff), (s["up"], s["x"], s["u"].data_ptr(), ff)], norm=s["norm"], silu=t == 1)
            s["last"] = fused([(s["down"], s["act"], s["out"].data_ptr(), n)], residual=s["x"])
        elif t > 8:
            s["ws"] = max((product_ws(c["type"], k, m, t) for k, m in ((n, ff), (ff, n))), key=lambda w: w.numel())
        return s

    @staticmethod
    def run(c, s):
        n, ff, t = c["width"], c["ff"], c["tokens"]
        if t <= 4:
            launch(c["type"], s["first"], n, ff, t)
            if t > 1:
                check(lib().b200_op_silu_mul(s["g"].data_ptr(), s["u"].data_ptr(), None, s["act"].data_ptr(), t * ff, None))
            launch(c["type_down"], s["last"], ff, n, t)
            return s["out"]
        check(lib().b200_op_rms_norm_mul(C.byref(tensor(s["x"], n, t)), s["norm"].data_ptr(), None, C.byref(tensor(s["h"], n, t)), EPS, None))
        if t <= 8:
            vector(c["type"], s["gate"], s["h"], s["g"], ff, n, t)
            vector(c["type"], s["up"], s["h"], s["u"], ff, n, t)
        else:
            product(c["type"], s["gate"], s["h"], s["g"], ff, n, t, s["ws"])
            product(c["type"], s["up"], s["h"], s["u"], ff, n, t, s["ws"], again=True)
        check(lib().b200_op_silu_mul(s["g"].data_ptr(), s["u"].data_ptr(), None, s["act"].data_ptr(), t * ff, None))
        if t <= 8:
            vector(c["type_down"], s["down"], s["act"], s["out"], n, ff, t)
        else:
            product(c["type_down"], s["down"], s["act"], s["out"], n, ff, t, s["ws"])
        return s["out"]

    @staticmethod
    def exact(c, seed):
        s = Mlp.weights(c, generator(seed))
        n, ff = c["width"], c["ff"]
        h = rms64(s["x"], s["norm"])
        act = silu64(h @ dequantised(s["gate"], c["type"], ff, n).T) * (h @ dequantised(s["up"], c["type"], ff, n).T)
        y = act @ dequantised(s["down"], c["type_down"], n, ff).T
        return y + s["x"] if c["tokens"] <= 4 else y

    @staticmethod
    def work(c):
        n, ff, t = c["width"], c["ff"], c["tokens"]
        return {"bytes": 2 * ff * row_bytes(c["type"], n) + n * row_bytes(c["type_down"], ff) + 4 * t * 2 * n, "flops": 6 * t * n * ff}


class Moe:
    @staticmethod
    def draw(rng):
        return {"width": 256 * spread(rng, 4, 16), "ff": 256 * spread(rng, 4, 40), "experts": rng.choice([4, 8, 8]), "used": rng.choice([1, 2, 2, 3]),
                "type": rng.choice(["q4_K", "q5_K", "q8_0", "q4_0"]), "type_down": rng.choice(["q6_K", "q4_K"]),
                "tokens": rng.choice([1, 1, 2, 4, 5]) if rng.random() < 0.5 else spread(rng, 9, 400)}

    @staticmethod
    def weights(c, g):
        n, ff, e, t = c["width"], c["ff"], c["experts"], c["tokens"]
        # a router's choice: some experts are asked for more often than others
        logits = normal(g, t, e) + normal(g, e, std=0.7)
        return {"gate": quantised(g, c["type"], e * ff, n), "up": quantised(g, c["type"], e * ff, n), "down": quantised(g, c["type_down"], e * n, ff),
                "h": activations(g, t, n) * 0.7, "ids": logits.topk(c["used"], dim=1).indices.int().contiguous()}

    @staticmethod
    def prepare(c, seed):
        s = Moe.weights(c, generator(seed))
        n, ff, t, used = c["width"], c["ff"], c["tokens"], c["used"]
        s["g"], s["u"], s["act"] = (torch.empty(t, used, ff, device="cuda") for _ in range(3))
        s["out"] = torch.empty(t, used, n, device="cuda")
        if t * used > 16:
            need = max(lib().b200_mul_mat_id_q_workspace_bytes(TYPES[c["type"]], k, m, used, t, c["experts"]) for k, m in ((n, ff), (ff, n)))
            s["ws"] = workspace(need)
        return s

    @staticmethod
    def experts(c, s, kind, w, x, rows_in, dst, k, m):
        t, used = c["tokens"], c["used"]
        rb = row_bytes(kind, k)
        head = (TYPES[kind], w.data_ptr(), rb, rb * m, c["experts"], s["ids"].data_ptr(), used, x.data_ptr(), k, rows_in * k, dst.data_ptr(), m, used * m, k, m, used, rows_in, t)
        if "ws" in s:
            check(lib().b200_mul_mat_id_q(*head, s["ws"].data_ptr(), s["ws"].numel(), None), "b200_mul_mat_id_q")
        else:
            check(lib().b200_mul_mat_id_vec_q(*head, None), "b200_mul_mat_id_vec_q")

    @staticmethod
    def run(c, s):
        n, ff, t, used = c["width"], c["ff"], c["tokens"], c["used"]
        Moe.experts(c, s, c["type"], s["gate"], s["h"], 1, s["g"], n, ff)
        Moe.experts(c, s, c["type"], s["up"], s["h"], 1, s["u"], n, ff)
        check(lib().b200_op_silu_mul(s["g"].data_ptr(), s["u"].data_ptr(), None, s["act"].data_ptr(), t * used * ff, None))
        Moe.experts(c, s, c["type_down"], s["down"], s["act"], used, s["out"], ff, n)
        return s["out"]

    @staticmethod
    def exact(c, seed):
        s = Moe.weights(c, generator(seed))
        n, ff = c["width"], c["ff"]
        out = torch.empty(c["tokens"], c["used"], n, dtype=torch.float64, device="cuda")

        def expert(name, kind, e, rows, k):
            size = rows * row_bytes(kind, k)
            return dequantised(s[name][e * size:(e + 1) * size], kind, rows, k)

        for e in range(c["experts"]):
            tok, slot = (s["ids"] == e).nonzero(as_tuple=True)
            if not len(tok):
                continue
            h = s["h"][tok].double()
            act = silu64(h @ expert("gate", c["type"], e, ff, n).T) * (h @ expert("up", c["type"], e, ff, n).T)
            out[tok, slot] = act @ expert("down", c["type_down"], e, n, ff).T
        return out

    @staticmethod
    def work(c):
        n, ff, pairs = c["width"], c["ff"], c["tokens"] * c["used"]
        per_expert = 2 * ff * row_bytes(c["type"], n) + n * row_bytes(c["type_down"], ff)
        return {"bytes": min(c["experts"], pairs) * per_expert + 4 * (c["tokens"] * n + pairs * n), "flops": 6 * pairs * n * ff}


class Attn:
    """Queries of `tokens` tokens behind `past` cached ones; the cache's rows hold all kv heads of a token, and the visible range is padded to 256 cells."""

    @staticmethod
    def draw(rng):
        group = rng.choice([1, 1, 4, 8])
        kv_heads = max(1, spread(rng, 8, 64) // group)
        tokens = rng.choice([1, 1, 1, 2, 4, 8]) if rng.random() < 0.5 else spread(rng, 16, 512)
        return {"heads": kv_heads * group, "kv_heads": kv_heads, "dim": rng.choice([64, 128, 128]), "kv": rng.choice(["f16", "f16", "q8_0"]), "tokens": tokens,
                "past": spread(rng, 1, 16000 if tokens == 1 else 2000)}

    @staticmethod
    def sizes(c):
        cells = -(-(c["past"] + c["tokens"]) // 256) * 256
        width = c["kv_heads"] * c["dim"]
        return cells, width, 2 * width if c["kv"] == "f16" else row_bytes("q8_0", width)

    @staticmethod
    def inputs(c, g):
        cells, width, rb = Attn.sizes(c)
        s = {"q": normal(g, c["heads"], c["tokens"], c["dim"], std=1.0)}
        for name in ("k", "v"):
            if c["kv"] == "f16":
                rows = normal(g, cells, width).half().view(torch.uint8)
            else:
                x = normal(g, cells, width // 32, 32)
                d = (x.abs().amax(dim=2, keepdim=True) / 127).half()
                q = torch.round(x / d.float()).clamp(-127, 127).to(torch.int8)
                rows = torch.cat([d.view(torch.uint8), q.view(torch.uint8)], dim=2)
            s[name] = torch.cat([rows.reshape(-1), torch.zeros(256, dtype=torch.uint8, device="cuda")])
        padded = -(-c["tokens"] // 64) * 64
        mask = torch.full((padded, cells), -math.inf, device="cuda", dtype=torch.float16)
        cell, tok = torch.arange(cells, device="cuda"), torch.arange(c["tokens"], device="cuda")
        mask[:c["tokens"]].masked_fill_(cell[None, :] <= c["past"] + tok[:, None], 0)
        s["mask"] = mask
        return s

    @staticmethod
    def prepare(c, seed):
        s = Attn.inputs(c, generator(seed))
        cells, width, rb = Attn.sizes(c)
        t, d = c["tokens"], c["dim"]
        s["out"] = torch.empty(t, c["heads"], d, device="cuda")
        head = rb // c["kv_heads"]
        kind = TYPES[c["kv"]]
        s["args"] = FattnArgs(s["q"].data_ptr(), s["k"].data_ptr(), s["v"].data_ptr(), s["mask"].data_ptr(), s["out"].data_ptr(), d, t, c["heads"], c["kv_heads"], cells, kind, kind,
                              4 * d, 4 * d * t, rb, head, rb, head, 2 * cells, d ** -0.5, 0.0, 0.0)
        s["ws"] = workspace(lib().b200_flash_attn_workspace_bytes(C.byref(s["args"])))
        return s

    @staticmethod
    def run(c, s):
        check(lib().b200_flash_attn_ext(C.byref(s["args"]), s["ws"].data_ptr(), s["ws"].numel(), None), "b200_flash_attn_ext")
        return s["out"]

    @staticmethod
    def rows64(c, flat):
        cells, width, rb = Attn.sizes(c)
        if c["kv"] == "f16":
            x = flat[:cells * rb].view(torch.float16).double()
        else:
            x = dequantised(flat, "q8_0", cells, width)
        return x.reshape(cells, c["kv_heads"], c["dim"])

    @staticmethod
    def exact(c, seed):
        s = Attn.inputs(c, generator(seed))
        k, v, mask = Attn.rows64(c, s["k"]), Attn.rows64(c, s["v"]), s["mask"][:c["tokens"]].double()
        out = torch.empty(c["tokens"], c["heads"], c["dim"], dtype=torch.float64, device="cuda")
        group = c["heads"] // c["kv_heads"]
        for h in range(c["heads"]):
            p = torch.softmax(s["q"][h].double() @ k[:, h // group].T * c["dim"] ** -0.5 + mask, dim=1)
            out[:, h] = p @ v[:, h // group]
        return out

    @staticmethod
    def work(c):
        cells, width, rb = Attn.sizes(c)
        t, seen = c["tokens"], c["past"] + c["tokens"]
        pairs = t * c["past"] + t * (t + 1) // 2
        return {"bytes": 2 * seen * rb + 8 * t * c["heads"] * c["dim"] + 2 * t * seen, "flops": 4 * pairs * c["heads"] * c["dim"]}


class Block:
    """The attention side of a layer in bf16 with f32 caches: a learned sink per head, optionally a window, the rows of `past` earlier tokens in the cache."""

    @staticmethod
    def draw(rng):
        group = rng.choice([1, 2, 4, 8])
        kv_heads = max(1, spread(rng, 8, 32) // group)
        tokens = tokens_of(rng)
        return {"width": 64 * spread(rng, 12, 64), "heads": kv_heads * group, "kv_heads": kv_heads, "dim": rng.choice([64, 128, 128]), "tokens": tokens,
                "past": spread(rng, 1, 1500), "window": rng.choice([0, 0, 300, 512])}

    @staticmethod
    def inputs(c, g):
        n, d, h, kv = c["width"], c["dim"], c["heads"], c["kv_heads"]
        seen = c["past"] + c["tokens"]
        cells = -(-seen // 256) * 256
        s = {"wqkv": normal(g, (h + 2 * kv) * d, n, std=n ** -0.5).bfloat16(), "wo": normal(g, n, h * d, std=(h * d) ** -0.5).bfloat16(), "x": normal(g, c["tokens"], n),
             "k": normal(g, cells, kv * d), "v": normal(g, cells, kv * d), "sink": normal(g, h)}
        at = torch.arange(cells, device="cuda", dtype=torch.int32)
        s["cell_pos"] = torch.where(at < seen, at, -1).int()
        s["cell_seq"] = torch.where(at < seen, 0, -1).int()
        s["pos"] = torch.arange(c["past"], seen, device="cuda", dtype=torch.int32)
        s["seq"] = torch.zeros(c["tokens"], device="cuda", dtype=torch.int32)
        s["freqs"] = (10000.0 ** (-torch.arange(0, d, 2, device="cuda").double() / d)).float()
        return s, cells

    @staticmethod
    def prepare(c, seed):
        s, cells = Block.inputs(c, generator(seed))
        n, d, h, kv, t = c["width"], c["dim"], c["heads"], c["kv_heads"], c["tokens"]
        m = (h + 2 * kv) * d
        s["qkv"], s["mix"], s["out"] = torch.empty(t, m, device="cuda"), torch.empty(t, h * d, device="cuda"), torch.empty(t, n, device="cuda")
        at = s["qkv"].data_ptr()
        s["store"] = QkvStoreArgs(q=at, q_stride=m, k=at + 4 * h * d, k_stride=m, v=at + 4 * (h + kv) * d, v_stride=m, pos=s["pos"].data_ptr(), cells=s["pos"].data_ptr(),
                                  freqs=s["freqs"].data_ptr(), k_cache=s["k"].data_ptr(), k_cache_stride=kv * d, v_cache=s["v"].data_ptr(), v_cache_stride=kv * d, n_head=h,
                                  n_head_kv=kv, dim=d, vdim=d, n_dims=d, n_tokens=t, eps=EPS)
        s["attend"] = SinkAttnArgs(q=at, q_stride=m, k_cache=s["k"].data_ptr(), k_cache_stride=kv * d, v_cache=s["v"].data_ptr(), v_cache_stride=kv * d,
                                   cell_seq=s["cell_seq"].data_ptr(), cell_pos=s["cell_pos"].data_ptr(), tok_seq=s["seq"].data_ptr(), tok_pos=s["pos"].data_ptr(),
                                   sink=s["sink"].data_ptr(), dst=s["mix"].data_ptr(), dst_stride=h * d, n_head=h, n_head_kv=kv, dim=d, vdim=d, n_tokens=t, n_kv=cells,
                                   window=c["window"], scale=d ** -0.5, bf16_products=1)
        s["need"] = int(lib().b200_sink_attn_workspace_bytes(C.byref(s["attend"])))
        s["aws"] = workspace(s["need"])
        if t > 8:
            s["ws"] = max((product_ws("bf16", a, b, t) for a, b in ((n, m), (h * d, n))), key=lambda w: w.numel())
        return s

    @staticmethod
    def dense(s, w, x, dst, rows, k, t):
        if t > 8:
            product("bf16", w, x, dst, rows, k, t, s["ws"])
        else:
            check(lib().b200_op_mul_mat_float(C.byref(tensor(w, k, rows, kind=BF16)), C.byref(tensor(x, k, t)), C.byref(tensor(dst, rows, t)), None), "b200_op_mul_mat_float")

    @staticmethod
    def run(c, s):
        n, d, h, kv, t = c["width"], c["dim"], c["heads"], c["kv_heads"], c["tokens"]
        Block.dense(s, s["wqkv"], s["x"], s["qkv"], (h + 2 * kv) * d, n, t)
        check(lib().b200_op_qkv_store(C.byref(s["store"]), None), "b200_op_qkv_store")
        check(lib().b200_op_sink_attn_ws(C.byref(s["attend"]), s["aws"].data_ptr(), s["need"], None), "b200_op_sink_attn_ws")
        Block.dense(s, s["wo"], s["mix"], s["out"], n, h * d, t)
        return [s["mix"], s["out"], s["k"], s["v"]]

    @staticmethod
    def exact(c, seed):
        s, cells = Block.inputs(c, generator(seed))
        d, h, kv, t = c["dim"], c["heads"], c["kv_heads"], c["tokens"]
        q, k, v = (s["x"].double() @ s["wqkv"].double().T).split([h * d, kv * d, kv * d], dim=1)
        angle = s["pos"].double()[:, None] * s["freqs"].double()[None, :]

        def turned(x):
            x = x.reshape(t, -1, d // 2, 2)
            co, si = torch.cos(angle)[:, None], torch.sin(angle)[:, None]
            return torch.stack([x[..., 0] * co - x[..., 1] * si, x[..., 0] * si + x[..., 1] * co], dim=-1).reshape(t, -1, d)

        kc, vc = s["k"].double(), s["v"].double()
        kc[c["past"]:c["past"] + t], vc[c["past"]:c["past"] + t] = turned(k).reshape(t, -1), v
        q, keys, values = turned(q), kc.reshape(cells, kv, d), vc.reshape(cells, kv, d)
        far = s["pos"][:, None] - s["cell_pos"][None, :]
        seen = (s["cell_seq"][None, :] == 0) & (far >= 0)
        if c["window"]:
            seen &= far < c["window"]
        mix = torch.empty(t, h, d, dtype=torch.float64, device="cuda")
        for i in range(h):
            score = (q[:, i] @ keys[:, i // (h // kv)].T * d ** -0.5).masked_fill(~seen, -math.inf)
            p = torch.softmax(torch.cat([score, s["sink"][i].double().expand(t, 1)], dim=1), dim=1)[:, :-1]
            mix[:, i] = p @ values[:, i // (h // kv)]
        mix = mix.reshape(t, h * d)
        return [mix, mix @ s["wo"].double().T, kc, vc]

    @staticmethod
    def work(c):
        n, d, h, kv, t = c["width"], c["dim"], c["heads"], c["kv_heads"], c["tokens"]
        seen = c["past"] + t
        weights = n * (2 * h + 2 * kv) * d
        reach = [min(c["window"] or seen, c["past"] + i + 1) for i in range(t)]
        rows = min(seen, (c["window"] or seen) + t)
        return {"bytes": 2 * weights + 4 * t * 2 * n + 4 * 2 * kv * d * (rows + t), "flops": 2 * t * weights + 4 * sum(reach) * h * d}


class Delta:
    @staticmethod
    def draw(rng):
        group = rng.choice([1, 1, 2])
        kv_heads = max(1, spread(rng, 4, 32) // group)
        many = rng.choice([1, 1, 1, 3, 8])
        return {"heads": kv_heads * group, "kv_heads": kv_heads, "dim": rng.choice([64, 128, 128]), "vdim": rng.choice([64, 128, 128]),
                "tokens": many * (1 if rng.random() < 0.3 else spread(rng, 2, 1024 // many)), "seqs": many, "per_channel": rng.random() < 0.5, "fresh": rng.random() < 0.5}

    @staticmethod
    def inputs(c, g):
        h, kv, d, vd, t = c["heads"], c["kv_heads"], c["dim"], c["vdim"], c["tokens"]
        channels = 2 * kv * d + h * vd
        gates = h * (d if c["per_channel"] else 1)
        s = {"x": normal(g, t, channels), "taps": normal(g, channels, 4, std=0.4), "a": normal(g, t, gates), "b": normal(g, t, h),
             "a_log": torch.log(1 + 15 * torch.rand(h, generator=g, device="cuda")), "dt": normal(g, gates) - 4.0,
             "start": normal(g, c["seqs"], h, vd, d, std=0.1), "before": normal(g, c["seqs"], 3, channels)}
        return s

    @staticmethod
    def prepare(c, seed):
        s = Delta.inputs(c, generator(seed))
        h, kv, d, vd, t, many = c["heads"], c["kv_heads"], c["dim"], c["vdim"], c["tokens"], c["seqs"]
        channels, each = 2 * kv * d + h * vd, t // many
        fresh = 1 if c["fresh"] else 0
        s["info"] = torch.tensor([[i * each for i in range(many)], [each] * many, list(range(many)), [fresh] * many], dtype=torch.int32, device="cuda")
        s["state"], s["tail"] = s["start"].clone(), s["before"].clone()
        s["y"], s["out"] = torch.empty(t, channels, device="cuda"), torch.empty(t, h * vd, device="cuda")
        s["conv"] = ShortConvArgs(x=s["x"].data_ptr(), x_stride=channels, w=s["taps"].data_ptr(), seq_info=s["info"].data_ptr(), n_seq=many, tail=s["tail"].data_ptr(),
                                  slot_stride=3 * channels, dst=s["y"].data_ptr(), dst_stride=channels, channels=channels, taps=4, act=1, n_tokens=t)
        at, gates = s["y"].data_ptr(), s["a"].shape[1]
        s["scan"] = DeltaRuleArgs(q=at, k=at + 4 * kv * d, v=at + 8 * kv * d, q_stride=channels, k_stride=channels, v_stride=channels, a=s["a"].data_ptr(), b=s["b"].data_ptr(),
                                  a_stride=gates, b_stride=h, a_log=s["a_log"].data_ptr(), dt_bias=s["dt"].data_ptr(), seq_info=s["info"].data_ptr(), n_seq=many,
                                  state=s["state"].data_ptr(), slot_stride=h * vd * d, dst=s["out"].data_ptr(), dst_stride=h * vd, heads=h, kv_heads=kv, dim=d, vdim=vd, unit_qk=1,
                                  unit_eps=1e-6, q_scale=d ** -0.5, channel_decay=1 if c["per_channel"] else 0)
        return s

    @staticmethod
    def run(c, s):
        check(lib().b200_op_short_conv(C.byref(s["conv"]), None), "b200_op_short_conv")
        check(lib().b200_op_delta_rule_scan(C.byref(s["scan"]), None), "b200_op_delta_rule_scan")
        return [s["out"], s["state"], s["tail"]]

    @staticmethod
    def exact(c, seed):
        s = Delta.inputs(c, generator(seed))
        h, kv, d, vd, many = c["heads"], c["kv_heads"], c["dim"], c["vdim"], c["seqs"]
        each = c["tokens"] // many
        x = s["x"].double().reshape(many, each, -1)
        before = torch.zeros_like(s["before"]).double() if c["fresh"] else s["before"].double()
        x = torch.cat([before, x], dim=1)
        y = silu64(sum(x[:, j:j + each] * s["taps"][:, j].double() for j in range(4)))
        q, k, v = (z.reshape(many, each, -1, w) for z, w in zip(y.split([kv * d, kv * d, h * vd], dim=2), (d, d, vd)))
        q, k = (torch.repeat_interleave(z / torch.sqrt(z.square().sum(-1, keepdim=True) + 1e-6), h // kv, dim=2) for z in (q, k))
        q = q * d ** -0.5
        soft = torch.nn.functional.softplus(s["a"].double() + s["dt"].double()).reshape(many, each, h, -1)
        keep = torch.exp(-torch.exp(s["a_log"].double())[:, None] * soft)[:, :, :, None, :]
        beta = torch.sigmoid(s["b"].double()).reshape(many, each, h, 1)
        state = torch.zeros_like(s["start"]).double() if c["fresh"] else s["start"].double()
        out = torch.empty(many, each, h, vd, dtype=torch.float64, device="cuda")
        for t in range(each):
            state = state * keep[:, t]
            u = beta[:, t] * (v[:, t] - (state * k[:, t, :, None, :]).sum(-1))
            state = state + u[..., None] * k[:, t, :, None, :]
            out[:, t] = (state * q[:, t, :, None, :]).sum(-1)
        return [out.reshape(c["tokens"], h * vd), state, x[:, each:]]

    @staticmethod
    def work(c):
        h, kv, d, vd, t = c["heads"], c["kv_heads"], c["dim"], c["vdim"], c["tokens"]
        channels, gates = 2 * kv * d + h * vd, h * (d if c["per_channel"] else 1)
        state = 4 * c["seqs"] * h * d * vd * (1 if c["fresh"] else 2)
        return {"bytes": 4 * t * (channels + gates + h + h * vd) + state, "flops": 7 * t * h * d * vd + 10 * t * channels}


class Model:
    """A greedy decoding loop of a Q4_0 / Q4_K_M decoder: `steps` calls with one token each behind `past` cached ones."""
    SHAPE = {"tiny": (2048, 22, 32, 4, 5632, 32000)}  # TinyLlama-1.1B: width, layers, heads, kv heads, ff, vocabulary

    @staticmethod
    def draw(rng):
        return {"shape": "tiny", "ftype": rng.choice(["Q4_0", "Q4_K_M"]), "kv": rng.choice(["f16", "f16", "q8_0"]), "past": spread(rng, 16, 1900), "steps": rng.choice([3, 5, 8])}

    @staticmethod
    def kinds(c):
        """(type, rows, values a row, gain) of every matrix.  The layers' results are small beside the stream, as in trained models."""
        n, layers, heads, kv_heads, ff, vocab = Model.SHAPE[c["shape"]]
        kv, branch = n // heads * kv_heads, 0.3
        base = "q4_0" if c["ftype"] == "Q4_0" else "q4_K"
        found = {"token_embd.weight": (base, vocab, n, 20.0), "output.weight": ("q6_K", vocab, n, 1.0)}
        for il in range(layers):
            # the layers of a _K_M mix whose v and down matrices have the larger type
            more = base == "q4_K" and (il < layers // 8 or il >= 7 * layers // 8 or (il - layers // 8) % 3 == 2)
            for leaf, rows, k, gain in (("attn_q", n, n, 1.0), ("attn_k", kv, n, 1.0), ("attn_v", kv, n, 1.0), ("attn_output", n, n, branch), ("ffn_gate", ff, n, 1.0),
                                        ("ffn_up", ff, n, 1.0), ("ffn_down", n, ff, branch)):
                found["blk.%d.%s.weight" % (il, leaf)] = ("q6_K" if more and leaf in ("attn_v", "ffn_down") else base, rows, k, gain)
        return found

    @staticmethod
    def inputs(c, seed):
        g = generator(seed)
        w = {name: quantised(g, *what) for name, what in Model.kinds(c).items()}
        return w, torch.randint(0, Model.SHAPE[c["shape"]][5], (c["steps"],), generator=g, device="cuda").tolist()

    @staticmethod
    def prepare(c, seed):
        n, layers, heads, kv_heads, ff, vocab = Model.SHAPE[c["shape"]]
        w, tokens = Model.inputs(c, seed)
        m = llama.LlamaModel(llama.ModelShape(c["shape"], n, layers, heads, kv_heads, ff, vocab, c["ftype"]), 2048, TYPES[c["kv"]])
        for name, (kind, rows, k, gain) in Model.kinds(c).items():
            m.set_tensor(name, TYPES[kind], (k, rows, 1), w[name][:rows * row_bytes(kind, k)].cpu().numpy())
        for name in ["output_norm.weight"] + ["blk.%d.%s.weight" % (il, leaf) for il in range(layers) for leaf in ("attn_norm", "ffn_norm")]:
            m.set_tensor(name, F32, (n, 1, 1), np.ones(n, dtype=np.float32))
        m.finalize(1)
        m.kv_fill_random(c["past"], seed=seed & 0xffff)
        return {"model": m, "tokens": tokens}

    @staticmethod
    def run(c, s):
        return [s["model"].decode([t], c["past"] + i)[0].copy() for i, t in enumerate(s["tokens"])]

    @staticmethod
    def exact(c, seed):
        n, layers, heads, kv_heads, ff, vocab = Model.SHAPE[c["shape"]]
        past, steps, d = c["past"], c["steps"], n // heads
        kv = kv_heads * d
        w, tokens = Model.inputs(c, seed)
        kinds = Model.kinds(c)

        def matrix(name):
            kind, rows, k, _ = kinds[name]
            return dequantised(w[name], kind, rows, k)

        x = np.random.default_rng(seed & 0xffff).standard_normal((past, kv), dtype=np.float32)
        if c["kv"] == "f16":
            x = x.astype(np.float16).astype(np.float64)
        else:
            b = x.reshape(past, kv // 32, 32)
            scale = (np.abs(b).max(axis=2, keepdims=True) / 127.0).astype(np.float32)
            x = (np.round(b / scale) * scale.astype(np.float16).astype(np.float64)).reshape(past, kv)
        cached = torch.from_numpy(x).cuda()
        at = torch.arange(past, past + steps, device="cuda").double()
        angle = (at[:, None] * 10000.0 ** (-torch.arange(0, d, 2, device="cuda").double() / d))[:, None]
        later = torch.arange(past + steps, device="cuda")[None, :] > at[:, None]

        def turned(z):
            z = z.reshape(steps, -1, d // 2, 2)
            return torch.stack([z[..., 0] * torch.cos(angle) - z[..., 1] * torch.sin(angle), z[..., 0] * torch.sin(angle) + z[..., 1] * torch.cos(angle)], dim=-1).reshape(steps, -1)

        x = matrix("token_embd.weight")[tokens]
        for il in range(layers):
            def layer(z, leaf):
                return z @ matrix("blk.%d.%s.weight" % (il, leaf)).T

            h = rms64(x)
            keys = torch.cat([cached, turned(layer(h, "attn_k"))]).reshape(-1, kv_heads, d)
            values = torch.cat([cached, layer(h, "attn_v")]).reshape(-1, kv_heads, d)
            q = turned(layer(h, "attn_q")).reshape(steps, kv_heads, heads // kv_heads, d)
            score = torch.einsum("tghd,cgd->tghc", q, keys) * d ** -0.5
            weight = torch.softmax(score.masked_fill(later[:, None, None, :], -math.inf), dim=-1)
            x = x + layer(torch.einsum("tghc,cgd->tghd", weight, values).reshape(steps, n), "attn_output")
            h = rms64(x)
            x = x + layer(silu64(layer(h, "ffn_gate")) * layer(h, "ffn_up"), "ffn_down")
        return list(rms64(x) @ matrix("output.weight").T)

    @staticmethod
    def work(c):
        n, layers, heads, kv_heads, ff, vocab = Model.SHAPE[c["shape"]]
        kv = n // heads * kv_heads
        matrices = [what for name, what in Model.kinds(c).items() if name != "token_embd.weight"]
        cache = 2 * layers * c["past"] * (2 * kv if c["kv"] == "f16" else row_bytes("q8_0", kv))
        weights = sum(rows * row_bytes(kind, k) for kind, rows, k, _ in matrices)
        flops = sum(2 * rows * k for _, rows, k, _ in matrices) + 4 * layers * c["past"] * n
        return {"bytes": c["steps"] * (weights + cache + 4 * vocab), "flops": c["steps"] * flops}


KINDS = {"proj": Proj, "mlp": Mlp, "moe": Moe, "attn": Attn, "block": Block, "delta": Delta, "model": Model}


# ------------------------------------------------------------------------------------------------ the cases
def listed():
    return [
        # the smallest calls: one token through the projections of a 1.1B Q4_0 decoder, a few microseconds a launch
        {"name": "proj_decode_1b", "kind": "proj", "width": 2048, "kv_width": 256, "type": "q4_0", "type_v": "q4_0", "tokens": 1},
        # most of a decoded token of a 7B Q4_K_M decoder
        {"name": "mlp_decode_7b", "kind": "mlp", "width": 4096, "ff": 11008, "type": "q4_K", "type_down": "q6_K", "tokens": 1},
        # four sequences decoded together, 13B Q5_K_M
        {"name": "mlp_decode_13b_batch4", "kind": "mlp", "width": 5120, "ff": 13824, "type": "q5_K", "type_down": "q6_K", "tokens": 4},
        # the 512-token batches in which a prompt is processed, 7B Q4_K_M
        {"name": "mlp_prompt_7b", "kind": "mlp", "width": 4096, "ff": 11008, "type": "q4_K", "type_down": "q6_K", "tokens": 512},
        # a short prompt of no round length, 13B Q5_K_M
        {"name": "proj_prompt_13b_ragged", "kind": "proj", "width": 5120, "kv_width": 5120, "type": "q5_K", "type_v": "q6_K", "tokens": 199},
        # routed experts over a prompt batch, Mixtral 8x7B Q4_K_M
        {"name": "moe_prompt_8x7b", "kind": "moe", "width": 4096, "ff": 14336, "experts": 8, "used": 2, "type": "q4_K", "type_down": "q6_K", "tokens": 512},
        # decoding at 4k context, 7B (every query head its own keys)
        {"name": "attn_decode_7b_4k", "kind": "attn", "heads": 32, "kv_heads": 32, "dim": 128, "kv": "f16", "tokens": 1, "past": 4000},
        # decoding at 32k context with a quantised cache, Mixtral 8x7B (four query heads share keys)
        {"name": "attn_decode_8x7b_32k_q8", "kind": "attn", "heads": 32, "kv_heads": 8, "dim": 128, "kv": "q8_0", "tokens": 1, "past": 32700},
        # the last batch of a 2k prompt, 7B
        {"name": "attn_prompt_7b_2k", "kind": "attn", "heads": 32, "kv_heads": 32, "dim": 128, "kv": "f16", "tokens": 512, "past": 1536},
        # a prompt batch through the attention side of a layer served from a folder
        {"name": "block_prompt_4096", "kind": "block", "width": 4096, "heads": 32, "kv_heads": 8, "dim": 128, "tokens": 512, "past": 512, "window": 0},
        # a prompt batch through the recurrent mixer of such a layer
        {"name": "delta_prompt_4096", "kind": "delta", "heads": 32, "kv_heads": 32, "dim": 128, "vdim": 128, "tokens": 512, "seqs": 1, "per_channel": False, "fresh": True},
        # whole calls, as a chat program makes them token by token
        {"name": "model_decode_1b", "kind": "model", "shape": "tiny", "ftype": "Q4_0", "kv": "f16", "past": 1000, "steps": 8},
    ]


def draw(rng):
    kind = rng.choice(list(KINDS))
    return {"kind": kind, **KINDS[kind].draw(rng)}


def prepare(case, seed):
    return case, KINDS[case["kind"]].prepare(case, seed)


def run(state):
    case, s = state
    return KINDS[case["kind"]].run(case, s)


def exact(case, seed):
    return KINDS[case["kind"]].exact(case, seed)


def work(case):
    return KINDS[case["kind"]].work(case)


def tolerance(case):
    """About four times what the path shows against 64 bits: q8_1 activations (8 bits a value under one scale per 32) when decoding, bf16
    operands for prompts, f16 scores and probabilities in attention over a cache, f32 throughout the delta rule."""
    kind, tokens = case["kind"], case.get("tokens", 1)
    if kind == "delta":
        return {"rel": 5e-6, "max": 1e-3}
    if kind == "attn":
        return {"rel": 2e-3, "max": 0.1}
    return {"rel": 1.5e-2 if kind != "model" and tokens > 8 else 3e-2, "max": 0.3}
