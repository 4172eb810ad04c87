"""The workloads this library is timed on: what its users have it do, through its public entry points.

Kinds of case:
  host     one drop-in operator call on host arrays (raster.quant.op): x up, y down, the call blocks
  linear   quantized matmuls on device buffers (Context.qmatmul), one call per matrix of the case
  decoder  one token through whole decoder layers, recorded once as a graph and replayed
  attn     decode attention of one token over a long cache
  train    a frozen-weight linear's forward and backward-data on device buffers
  load     a dense matrix quantized and bound (raster.quant.core), as a model loader does per matrix

`a`, `b` of a case: the [out, in] of its first and second matrix (the second one is absent when b_out is 0).
The weights are N(0, 0.02) or N(0, 0.015) quantized per block, the activations N(0, 1).
"""
import math

import numpy as np
import torch

from raster_b200 import _lib as L
from raster_b200.quant import core, cpu_quant, op
from raster_b200.runtime import default_context

FMT = {"q4_0": L.FMT_Q4_0, "q8_0": L.FMT_Q8_0, "q8_s": L.FMT_Q8_S}
KQUANT = ("q4_K", "q6_K")


def listed():
    return [
        # the reference's own host-array operator at one attention projection: the latency of a drop-in call
        {"name": "host_call_q8_4096x4096", "kind": "host", "fmt": "q8_0", "a_out": 4096, "a_in": 4096},
        # a 7B-class model's MLP at one token, called directly: the plainest decode step
        linear("mlp7b_q4_m1", "q4_0", 11008, 4096, 4096, 11008, 1, "a8", "f32", "f32"),
        # the same MLP for a small batch of sequences
        linear("mlp7b_q4_m8", "q4_0", 11008, 4096, 4096, 11008, 8, "a8", "f32", "f32"),
        # the same MLP in the mixed super-block formats models are published in
        linear("mlp7b_q4k_q6k_m1", "q4_K+q6_K", 11008, 4096, 4096, 11008, 1, "a8", "f32", "f32"),
        # a 70B-class MLP for a batch of 16 sequences, bf16 activations as they are
        linear("mlp70b_q4_m16_bf16", "q4_0", 28672, 8192, 8192, 28672, 16, "f", "bf16", "f32"),
        # the whole decode step around the matmuls: four 7B-class layers, one token, 1024 cached positions
        {"name": "decoder7b_q4_len1024", "kind": "decoder", "bits": 4, "layers": 4, "hidden": 4096, "ffn": 11008,
         "n_q": 32, "n_kv": 32, "head_dim": 128, "cache_len": 1024},
        # grouped-query attention late in a long conversation
        {"name": "attn_32q_8kv_len4096", "kind": "attn", "n_q": 32, "n_kv": 8, "head_dim": 128, "cache_len": 4096},
        # prefill of one projection, bf16 in and out
        linear("prefill_q8_m512", "q8_0", 4096, 4096, 0, 0, 512, "f", "bf16", "bf16"),
        # a short prompt whose sizes are no multiple of any tile, in the quantized-activation arithmetic
        linear("prompt_ragged_q4_m100", "q4_0", 11000, 4128, 0, 0, 100, "a8", "f32", "f32"),
        # prefill of a 70B-class MLP: the largest
        linear("prefill70b_q4_m256", "q4_0", 28672, 8192, 8192, 28672, 256, "f", "bf16", "f32"),
        # fine-tuning adapters over a frozen int8 linear: forward and backward-data of a batch of tokens
        {"name": "train_q8_m512", "kind": "train", "a_out": 4096, "a_in": 4096, "m": 512},
        # loading a model: one projection quantized and bound
        {"name": "load_q4_4096x4096", "kind": "load", "fmt": "q4_0", "a_out": 4096, "a_in": 4096},
    ]


def linear(name, fmt, a_out, a_in, b_out, b_in, m, mode, act, out):
    c = {"name": name, "kind": "linear", "fmt": fmt, "a_out": a_out, "a_in": a_in, "b_out": b_out, "b_in": b_in, "m": m,
         "mode": mode, "act": act, "out": out}
    return c


def logint(rng, lo, hi, step=1):
    """A multiple of `step` in [lo, hi], spread over its logarithm."""
    v = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi))) / step)) * step
    return min(max(v, -(-lo // step) * step), hi // step * step)


def draw(rng):
    kind = rng.choice(["host", "linear", "linear", "linear", "linear", "prefill", "prefill", "decoder", "attn", "train",
                       "load"])
    if kind == "host":
        return {"kind": "host", "fmt": rng.choice(["q4_0", "q8_0"]), "a_out": logint(rng, 1024, 11008, 8),
                "a_in": logint(rng, 1024, 11008, 32)}
    if kind == "linear":        # decode: 1 .. 16 tokens
        fmt = rng.choice(["q4_0", "q4_0", "q8_0", "q4_K", "q6_K"])
        kq = fmt in KQUANT
        mode = "a8" if kq else rng.choice(["a8", "a8", "f"])
        a_in = logint(rng, 1024, 28672, 256 if kq else 32)
        a_out = logint(rng, 1000, min(28672, 28672 * 8192 // a_in), 8)
        b_in = logint(rng, 1024, 16384, 256 if kq else 32)
        b_out = logint(rng, 1000, min(28672, 28672 * 4096 // b_in), 8)
        c = linear("", fmt, a_out, a_in, b_out, b_in, logint(rng, 1, 16), mode,
                   "f32" if kq else rng.choice(["f32", "bf16"]), "f32")
    elif kind == "prefill":     # a prompt of 17 .. 2048 tokens
        mode = rng.choice(["f", "f", "a8"])
        m = logint(rng, 17, 2048)
        cap = min(28672 * 8192, 60 * 10 ** 9 // m)
        a_in = logint(rng, 1024, min(16384, cap // 1000), 32)
        a_out = logint(rng, 1000, min(28672, cap // a_in), 8)
        c = linear("", rng.choice(["q4_0", "q8_0"]), a_out, a_in, 0, 0, m, mode, rng.choice(["f32", "bf16"]),
                   rng.choice(["f32", "bf16"]))
    elif kind == "decoder":
        n_kv, group = rng.choice([(32, 1), (8, 4), (16, 2), (16, 1), (4, 8)])
        return {"kind": "decoder", "bits": rng.choice([4, 8]), "layers": rng.randint(1, 3), "hidden": n_kv * group * 128,
                "ffn": logint(rng, 5632, 14336, 256), "n_q": n_kv * group, "n_kv": n_kv, "head_dim": 128,
                "cache_len": logint(rng, 32, 4096)}
    elif kind == "attn":
        n_kv, group = rng.choice([(8, 4), (8, 8), (32, 1), (4, 7), (16, 2)])
        hd = rng.choice([128, 128, 64])
        return {"kind": "attn", "n_q": n_kv * group, "n_kv": n_kv, "head_dim": hd,
                "cache_len": logint(rng, 128, min(32768, 4194304 // n_kv // hd))}
    elif kind == "train":
        m = logint(rng, 16, 2048)
        a_in = logint(rng, 1024, 8192, 32)
        return {"kind": "train", "a_out": logint(rng, 1024, min(11008, 30 * 10 ** 9 // m // a_in), 8), "a_in": a_in, "m": m}
    else:
        a_in = logint(rng, 1024, 4096, 256)
        return {"kind": "load", "fmt": rng.choice(["q4_0", "q8_0", "q4_K", "q6_K"]), "a_in": a_in,
                "a_out": logint(rng, 256, (8 << 20) // a_in, 8)}
    del c["name"]
    return c


def gen_of(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def normal(gen, *shape, sigma=1.0):
    return torch.randn(*shape, generator=gen, device="cuda") * sigma


def round_up_half(v):
    return torch.floor(v + 0.5)


def nibbles(q):
    """[..., 32] codes -> element k low, element k + 16 high nibble."""
    q = q.to(torch.uint8).reshape(-1, 32)
    return q[:, :16] | (q[:, 16:] << 4)


def quantized(gen, fmt, out, in_, sigma):
    """A matrix of N(0, sigma) in the arrays of its format, on the device."""
    w = normal(gen, out, in_, sigma=sigma)
    if fmt in ("q4_0", "q8_0"):
        zp, top = (8, 15) if fmt == "q4_0" else (128, 255)
        w = w.reshape(-1, 32)
        v = w.gather(1, w.abs().argmax(1, keepdim=True))
        d = v / -zp
        q = torch.clamp(round_up_half(w / d) + zp, 0, top)
        return {"wq": nibbles(q) if fmt == "q4_0" else q.to(torch.uint8), "ws": d}
    if fmt == "q8_s":
        w = w.reshape(-1, 32)
        d = w.abs().amax(1, keepdim=True) / 127
        return {"wq": torch.clamp(round_up_half(w / d), -127, 127).to(torch.int8), "ws": d}
    if fmt == "q4_K":
        w = w.reshape(-1, 8, 32)
        a, b = (w.amax(2) - w.amin(2)) / 15, w.amin(2)
        da, db = a.amax(1, keepdim=True) / 63, b.abs().amax(1, keepdim=True) / 31
        aq, bq = torch.clamp(round_up_half(a / da), 1, 63), torch.clamp(round_up_half(b / db), -32, 31)
        q = torch.clamp(round_up_half((w - (db * bq)[:, :, None]) / (da * aq)[:, :, None]), 0, 15)
        return {"wq": nibbles(q), "da": da, "db": db, "aq": aq.to(torch.int8), "bq": bq.to(torch.int8)}
    w = w.reshape(-1, 16, 16)
    a = w.abs().amax(2) / 32
    ds = a.amax(1, keepdim=True) / 127
    sc = torch.clamp(round_up_half(a / ds), 1, 127)
    q = torch.clamp(round_up_half(w / (ds * sc)[:, :, None]) + 32, 0, 63)
    return {"wq": q.to(torch.uint8), "sc": sc.to(torch.int8), "ds": ds}


def on_host(arrays):
    return {k: v.contiguous().cpu().numpy().ravel() for k, v in arrays.items()}


def bind(ctx, fmt, arrays, out, in_):
    h = on_host(arrays)
    if fmt == "q4_K":
        return ctx.bind_weight_q4k(h, out, in_)
    if fmt == "q6_K":
        return ctx.bind_weight_q6k(h, out, in_)
    return ctx.bind_weight(h["wq"], h["ws"], out, in_, FMT[fmt], L.LAYOUT_ROWMAJOR)


class State:
    """What a program of the case's kind holds; the library's handles are released with it."""

    def __init__(self, case, seed):
        self.case, self.ctx, self.gen = case, default_context(), gen_of(seed)
        self.handles, self.graph, self.tensors = [], None, []

    def weight(self, fmt, arrays, out, in_):
        self.handles.append(bind(self.ctx, fmt, arrays, out, in_))
        return self.handles[-1]

    def buffer(self, tensor):
        """The library's handle on a tensor's memory."""
        self.tensors.append(tensor)
        dt = {torch.float32: np.float32, torch.bfloat16: np.uint16, torch.int8: np.int8, torch.int32: np.int32,
              torch.int64: np.int64}[tensor.dtype]
        self.handles.append(self.ctx.wrap_buffer(tensor.data_ptr(), tensor.numel(), dt))
        return self.handles[-1]

    def zeros(self, *shape, dtype=torch.float32):
        t = torch.zeros(*shape, dtype=dtype, device="cuda")
        return t, self.buffer(t)

    def __del__(self):
        if self.graph is not None:
            self.graph.destroy()
        for h in reversed(self.handles):
            h.free()


def prepare(case, seed):
    s = State(case, seed)
    globals()["prepare_" + case["kind"]](s, case)
    torch.cuda.synchronize()
    return s


def run(s):
    return globals()["run_" + s.case["kind"]](s)


# ---- one operator call on host arrays ----
def prepare_host(s, c):
    q = on_host(quantized(s.gen, c["fmt"], c["a_out"], c["a_in"], 0.02))
    s.w = cpu_quant.repack_stream(q["wq"], q["ws"], c["a_out"], c["a_in"], cpu_quant.q4_0 if c["fmt"] == "q4_0" else cpu_quant.q8_0)
    s.x = normal(s.gen, c["a_in"]).cpu().numpy()
    s.y = np.empty(c["a_out"], dtype=np.float32)
    s.call = op.qlinear_i8_into if c["fmt"] == "q4_0" else op.qlinear_i8_q8_into
    run_host(s)     # the matrix goes to the device at the first call that sees it


def run_host(s):
    c = s.case
    return s.call(s.x, s.w["wqi"], s.w["wsi"], s.y, c["a_in"], c["a_out"])


# ---- matmuls on device buffers ----
def prepare_linear(s, c):
    dt = {"f32": torch.float32, "bf16": torch.bfloat16}
    fmts = c["fmt"].split("+")
    s.calls, s.outputs = [], []
    for i, (out, in_) in enumerate(((c["a_out"], c["a_in"]), (c["b_out"], c["b_in"]))):
        if out:
            fmt = fmts[i % len(fmts)]
            w = s.weight(fmt, quantized(s.gen, fmt, out, in_, 0.02 if in_ < 8192 else 0.015), out, in_)
            x = s.buffer(normal(s.gen, c["m"], in_).to(dt[c["act"]]))
            y, by = s.zeros(c["m"], out, dtype=dt[c["out"]])
            s.calls.append((w, x, by))
            s.outputs.append(y)
    code = {"f32": L.F32, "bf16": L.BF16}
    s.how = (c["m"], code[c["act"]], code[c["out"]], L.MODE_A8 if c["mode"] == "a8" else L.MODE_F)


def run_linear(s):
    for w, x, y in s.calls:
        s.ctx.qmatmul(w, x, y, *s.how)
    return s.outputs


# ---- one token through decoder layers, as a recorded graph ----
def prepare_decoder(s, c):
    H, F, NQ, NKV, HD, clen = c["hidden"], c["ffn"], c["n_q"], c["n_kv"], c["head_dim"], c["cache_len"]
    ctx, kv, fmt = s.ctx, NKV * HD, "q4_0" if c["bits"] == 4 else "q8_0"
    stack, s.caches = [], []
    for _ in range(c["layers"]):
        lay = {}
        for name, out, in_ in (("qkv", H + 2 * kv, H), ("o", H, H), ("gate_up", 2 * F, H), ("down", H, F)):
            lay[name] = s.weight(fmt, quantized(s.gen, fmt, out, in_, 0.02), out, in_)
        for name in ("kc", "vc"):
            s.caches.append(normal(s.gen, clen, kv))
            lay[name] = s.buffer(s.caches[-1])
        for name in ("n1", "n2"):
            lay[name] = s.buffer(1 + 0.1 * normal(s.gen, H))
        stack.append(lay)
    emb, nothing = s.buffer(normal(s.gen, H)), s.zeros(H)[1]
    s.x, x = s.zeros(H)
    s.down, down = s.zeros(H)
    h, o_, att = (s.zeros(H)[1] for _ in range(3))
    qkv = s.zeros(H + 2 * kv)[0]
    q, k, v = (s.buffer(t) for t in (qkv[:H], qkv[H:H + kv], qkv[H + kv:]))
    gu = s.zeros(2 * F)[0]
    g, u, bqkv, bgu = s.buffer(gu[:F]), s.buffer(gu[F:]), s.buffer(qkv), s.buffer(gu)
    xq, xs, xsum = s.zeros(H, dtype=torch.int8)[1], s.zeros(H // 32)[1], s.zeros(H // 32, dtype=torch.int32)[1]
    aq, as_, asum = s.zeros(F, dtype=torch.int8)[1], s.zeros(F // 32)[1], s.zeros(F // 32, dtype=torch.int32)[1]
    pos = s.buffer(torch.tensor([clen - 1], dtype=torch.int64, device="cuda"))
    length = s.buffer(torch.tensor([clen], dtype=torch.int64, device="cuda"))

    def step():
        for i, lay in enumerate(stack):
            ctx.residual_rms_norm_quant_act(x if i else emb, down if i else nothing, h, lay["n1"], xq, xs, xsum, 1, H)
            ctx.qmatmul_prequant(lay["qkv"], xq, xs, xsum, bqkv, 1)
            ctx.rope_append(q, k, v, lay["kc"], lay["vc"], NQ, NKV, HD, 10000.0, maxpos=clen, posbuf=pos)
            ctx.gqa_decode_attention_quant_act(q, lay["kc"], lay["vc"], att, xq, xs, xsum, 0, NQ, NQ // NKV, NKV, HD, clen,
                                               HD ** -0.5, clenbuf=length)
            ctx.qmatmul_prequant(lay["o"], xq, xs, xsum, o_, 1)
            ctx.residual_rms_norm_quant_act(h, o_, x, lay["n2"], xq, xs, xsum, 1, H)
            ctx.qmatmul_prequant(lay["gate_up"], xq, xs, xsum, bgu, 1)
            ctx.silu_mul_quant_act(g, u, aq, as_, asum, F)
            ctx.qmatmul_prequant(lay["down"], aq, as_, asum, down, 1)

    torch.cuda.synchronize()
    step()
    ctx.sync()
    ctx.graph_begin()
    step()
    s.graph = ctx.graph_end()


def run_decoder(s):
    s.graph.replay()
    return [s.x, s.down] + s.caches


# ---- decode attention ----
def prepare_attn(s, c):
    rows = c["n_kv"] * c["head_dim"]
    q = s.buffer(normal(s.gen, c["n_q"] * c["head_dim"]))
    k, v = s.buffer(normal(s.gen, c["cache_len"], rows)), s.buffer(normal(s.gen, c["cache_len"], rows))
    s.out, out = s.zeros(c["n_q"] * c["head_dim"])
    s.args = (q, k, v, out, c["cache_len"], c["n_q"], c["n_q"] // c["n_kv"], c["n_kv"], c["head_dim"], c["cache_len"],
              c["head_dim"] ** -0.5)


def run_attn(s):
    s.ctx.gqa_decode_attention(*s.args)
    return s.out


# ---- forward and backward-data of a frozen int8 linear ----
def prepare_train(s, c):
    q = quantized(s.gen, "q8_s", c["a_out"], c["a_in"], 0.02)
    s.w = s.weight("q8_s", q, c["a_out"], c["a_in"])
    s.codes, s.scales = s.buffer(q["wq"]), s.buffer(q["ws"])
    s.x, s.dy = s.buffer(normal(s.gen, c["m"], c["a_in"])), s.buffer(normal(s.gen, c["m"], c["a_out"], sigma=1e-3))
    (s.y, s.by), (s.dx, s.bdx) = s.zeros(c["m"], c["a_out"]), s.zeros(c["m"], c["a_in"])


def run_train(s):
    c = s.case
    s.ctx.qmatmul(s.w, s.x, s.by, c["m"], L.F32, L.F32, L.MODE_F)
    s.ctx.qlinear_q8_dx_device(s.dy, s.codes, s.scales, s.bdx, c["m"], c["a_in"], c["a_out"])
    return [s.y, s.dx]


# ---- a matrix quantized and bound, then used once ----
def prepare_load(s, c):
    s.w = normal(s.gen, c["a_out"], c["a_in"], sigma=0.02).cpu().numpy()
    s.x = normal(s.gen, c["a_in"]).cpu().numpy()
    s.bound = None


def run_load(s):
    c = s.case
    if s.bound is not None:     # the matrix this one takes the place of
        s.bound.free()
    qm = core.qmatrix(c["fmt"], s.w, c["a_out"], c["a_in"])
    s.bound = qm.data["bound"]
    s.handles = [s.bound]
    return {"y": core.matmul(qm, s.x), **{k: v for k, v in qm.data.items() if k != "bound"}}


# ---- what a pass cannot do without ----
def weight_bytes(fmt, out, in_):
    per = {"q4_0": 0.5 + 4 / 32, "q8_0": 1 + 4 / 32, "q8_s": 1 + 4 / 32, "q4_K": 0.5 + 8 / 256 + 2 / 32,
           "q6_K": 1 + 1 / 16 + 4 / 256}
    return out * in_ * per[fmt]


def work(c):
    size = {"f32": 4, "bf16": 2}
    if c["kind"] == "host":
        return {"bytes": weight_bytes(c["fmt"], c["a_out"], c["a_in"]) + 4 * (c["a_in"] + c["a_out"]),
                "flops": 2 * c["a_out"] * c["a_in"]}
    if c["kind"] == "linear":
        fmts, b, f = c["fmt"].split("+"), 0, 0
        for i, (out, in_) in enumerate(((c["a_out"], c["a_in"]), (c["b_out"], c["b_in"]))):
            if out:
                b += weight_bytes(fmts[i % len(fmts)], out, in_) + c["m"] * (in_ * size[c["act"]] + out * size[c["out"]])
                f += 2 * c["m"] * out * in_
        return {"bytes": b, "flops": f}
    if c["kind"] == "decoder":
        H, kv, fmt = c["hidden"], c["n_kv"] * c["head_dim"], "q4_0" if c["bits"] == 4 else "q8_0"
        n = (H + 2 * kv) * H + H * H + 3 * H * c["ffn"]
        return {"bytes": c["layers"] * (weight_bytes(fmt, n, 1) + 8 * c["cache_len"] * kv),
                "flops": c["layers"] * (2 * n + 4 * c["cache_len"] * c["n_q"] * c["head_dim"])}
    if c["kind"] == "attn":
        return {"bytes": 8 * c["cache_len"] * c["n_kv"] * c["head_dim"] + 8 * c["n_q"] * c["head_dim"],
                "flops": 4 * c["cache_len"] * c["n_q"] * c["head_dim"]}
    n = c["a_out"] * c["a_in"]
    if c["kind"] == "train":
        return {"bytes": 2 * weight_bytes("q8_s", n, 1) + 8 * c["m"] * (c["a_out"] + c["a_in"]), "flops": 4 * c["m"] * n}
    return {"bytes": 4 * n + weight_bytes(c["fmt"], n, 1), "flops": 2 * n}


def tolerance(c):
    if c["kind"] == "linear":
        if c["out"] == "bf16":
            return {"rel": 5e-3}                 # results rounded to 8 bits
        if c["m"] >= (64 if c["mode"] == "a8" else 17):
            return {"rel": 1e-3}                 # the prefill path multiplies 11-bit operands (documented: 1e-3)
        if c["mode"] == "f" and c["m"] > 1:
            return {"rel": 1e-3 if c["m"] > 8 and c["act"] == "f32" else 2e-5}   # f32 activations above 8 tokens: the same
        return {"rel": 1e-5, "max": 1e-4}
    if c["kind"] == "decoder":
        return {"rel": 2e-3, "max": 5e-2}        # an activation next to a rounding boundary may take the next 8-bit code
    if c["kind"] == "train":
        return {"rel": 1e-3}                     # the forward's operands have 11 bits
    if c["kind"] == "load":
        return {"rel": 1e-5, "max": 1e-4, "differ": 0.0}
    return {"rel": 1e-5, "max": 1e-4}
