"""Performance cases of the quantized-matmul backend: what its users have it do, through the calls they make.

Every case is a dict of plain values.  `op` says which calls a pass consists of:
  calls     one qmatmul per layer, one after another (a program that goes through its layers by itself)
  token     a decoder layer's seven projections and two rms-norms, one call each, every call fed by an earlier one
  batch     independent decode matmuls of one shape handed over in one qmatmul_batch call
  chain     a decode step through several layers, recorded once and replayed as a graph
  requant   weights quantized from fp32 (encode) and expanded again (decode)
Weights, scales, biases, activations, output buffers and the recorded graph are what such a program keeps; a pass is the
calls alone.  Layers of a case have weights of their own, so that a pass streams them instead of finding the last one
in a cache, as in a model larger than L2.
"""
import math

import torch

import mlx_b200
from mlx_b200.plugin import BF16, F32, PRO_RMS_NORM, PRO_SUM3

EPS = 1e-6
DTYPES = {"bf16": (torch.bfloat16, BF16), "f32": (torch.float32, F32)}
MATMUL = {"bits": 4, "group": 64, "dtype": "bf16", "out": "bf16"}


def listed():
    return [
        # one small layer, one row: nothing but the latency of a call
        dict(MATMUL, name="small_call", op="calls", M=1, K=1024, N=1024, layers=1),
        # one token of a 4096-wide decoder at batch 1, call by call
        dict(MATMUL, name="token_calls_m1", op="token", M=1, K=4096, N=11008, layers=2),
        # the decode sweep: 12 layers at each of four batch sizes
        dict(MATMUL, name="decode_sweep_batch", op="batch", rows="1,4,8,16", K=4096, N=11008, layers=48),
        # one decode step at batch 8, recorded as a graph
        dict(MATMUL, name="decode_chain_graph_m8", op="chain", M=8, K=4096, N=11008, layers=4),
        # a large 8-bit output layer at the largest decode batch
        dict(MATMUL, name="decode_8bit_m16", op="calls", M=16, K=8192, N=28672, layers=1, bits=8, group=128),
        # widths that are no power of two and a vocabulary-like odd number of rows
        dict(MATMUL, name="decode_ragged_m3", op="calls", M=3, K=2880, N=5003, layers=8),
        # short prompts or many requests at once: more rows than decode takes, far fewer than a prefill tile
        dict(MATMUL, name="short_prefill_m48", op="calls", M=48, K=4096, N=11008, layers=4),
        # prefill of 2048 tokens, 4 bits
        dict(MATMUL, name="prefill_4bit_m2048", op="calls", M=2048, K=4096, N=4096, layers=1),
        # the large 8-bit layer at 512 tokens
        dict(MATMUL, name="prefill_8bit_m512", op="calls", M=512, K=8192, N=28672, layers=1, bits=8, group=128),
        # a prompt of no particular length on a layer of no particular width
        dict(MATMUL, name="prefill_ragged_m777", op="calls", M=777, K=2880, N=5003, layers=2, group=32),
        # full precision: fp32 activations, scales and biases, one row
        dict(MATMUL, name="fp32_m1", op="calls", M=1, K=4096, N=4096, layers=8, dtype="f32", out="f32"),
        # a layer's weights on their way into the format and back
        dict(MATMUL, name="requant_4bit", op="requant", K=4096, N=11008, layers=1),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _draw(rng):
    op = rng.choice(["calls", "calls", "calls", "prefill", "prefill", "fp32", "token", "batch", "batch", "chain", "requant"])
    group, bits = rng.choice([32, 64, 64, 128]), rng.choice([4, 4, 8])
    block = max(group, 1024 // bits)
    c = dict(MATMUL, op="calls", bits=bits, group=group, layers=1)
    if op == "calls":     # decode: any width that the format has, any number of rows
        unit = rng.choice([group, block])
        c.update(M=_log(rng, 1, 16), K=unit * max(1, _log(rng, 512, 16384) // unit), N=_log(rng, 256, 32768), layers=rng.randint(1, 8),
                 out=rng.choice(["bf16", "bf16", "f32"]))
    elif op == "prefill":
        c.update(M=_log(rng, 17, 4096), K=128 * max(4, _log(rng, 512, 11008) // 128), N=_log(rng, 256, 28672), layers=rng.randint(1, 2))
        if group < 128:
            c["K"] += 64 * rng.randint(0, 1)
    elif op == "fp32":
        c.update(M=_log(rng, 1, 32), K=group * max(1, _log(rng, 512, 8192) // group), N=_log(rng, 256, 8192), layers=rng.randint(1, 8),
                 dtype="f32", out="f32")
    elif op == "batch":
        c.update(op="batch", K=block * max(1, _log(rng, 1024, 8192) // block), N=_log(rng, 512, 12288), layers=rng.randint(4, 48),
                 rows=",".join(str(_log(rng, 1, 16)) for _ in range(rng.randint(1, 4))))
    elif op in ("token", "chain"):
        c.update(op=op, M=_log(rng, 1, 8), K=block * max(2, _log(rng, 1024, 2 * 2048 if bits == 4 else 2048) // block),
                 N=block * max(2, _log(rng, 2048, 11008) // block), layers=rng.randint(1, 4))
    else:
        c.update(op="requant", K=group * max(1, _log(rng, 512, 11008) // group), N=_log(rng, 256, 12288), dtype=rng.choice(["bf16", "f32"]))
    return c


def _cost(case):
    w = work(case)
    return max(w["bytes"] / 6.4e12, w["flops"] / (1.7e15 if case["dtype"] == "bf16" else 7e13))


def draw(rng):
    most = max(_cost(c) for c in listed())
    while True:
        c = _draw(rng)
        if _cost(c) <= most:
            return c


def _rows(case):
    """Rows of x of every matmul of a batch."""
    ms = [int(m) for m in case["rows"].split(",")]
    return [ms[i % len(ms)] for i in range(case["layers"])]


def _projections(case):
    """(name, N, K) of a decoder layer: K is its width, N its inner width."""
    d, f = case["K"], case["N"]
    if case["op"] == "token":
        return [("q", d, d), ("k", d, d), ("v", d, d), ("o", d, d), ("gate", f, d), ("up", f, d), ("down", d, f)]
    return [("qkv", 3 * d, d), ("o", d, d), ("gateup", 2 * f, d), ("down", d, f)]


def _layer_bytes(case, K, N):
    return N * K * case["bits"] // 8 + 2 * N * (K // case["group"]) * (2 if case["dtype"] == "bf16" else 4)


def work(case):
    n = case["layers"]
    if case["op"] == "requant":  # fp32 weights in, packed words, scales and biases out; and those in, weights out
        N, K = case["N"], case["K"]
        return {"bytes": N * K * 4 + 2 * _layer_bytes(case, K, N) + N * K * (2 if case["dtype"] == "bf16" else 4), "flops": 6 * N * K}
    if case["op"] in ("token", "chain"):
        ps = _projections(case)
        act = case["M"] * 2 * sum(N + K for _, N, K in ps)
        return {"bytes": n * (sum(_layer_bytes(case, K, N) for _, N, K in ps) + act), "flops": n * 2 * case["M"] * sum(N * K for _, N, K in ps)}
    N, K = case["N"], case["K"]
    rows = sum(_rows(case)) if case["op"] == "batch" else n * case["M"]
    xs, ys = (2 if case["dtype"] == "bf16" else 4), (2 if case["out"] == "bf16" else 4)
    return {"bytes": n * _layer_bytes(case, K, N) + rows * (K * xs + N * ys), "flops": 2 * rows * N * K}


def tolerance(case):
    if case["op"] == "requant":
        return "exact"
    if case["op"] in ("token", "chain"):  # bf16 activations rounded anew in each of the steps
        return {"rel": 1e-2, "max": 8e-2}
    if case["out"] == "bf16":             # one rounding to bf16 at the end of an fp32 sum
        return {"rel": 4e-3, "max": 1.6e-2}
    return {"rel": 1e-5, "max": 2e-4}     # fp32 sums of up to 16384 products


class _State:
    """Tensors and the plugin's handles to them."""

    def __init__(self, case, ctx, seed):
        self.case, self.ctx, self.tensors, self.handles, self.graph = case, ctx, [], [], None
        self.gen = torch.Generator(device="cuda").manual_seed(seed)

    def wrap(self, t):
        b = self.ctx.wrap(t.data_ptr(), t.numel() * t.element_size(), tuple(t.shape))
        self.tensors.append(t)
        self.handles.append(b)
        return b

    def empty(self, shape, dtype):
        t = torch.empty(shape, dtype=dtype, device="cuda")
        return t, self.wrap(t)

    def normal(self, shape, dtype, std=1.0):
        return torch.randn(shape, generator=self.gen, device="cuda").mul_(std).to(dtype)

    def layer(self, N, K):
        """Packed words over the whole code range, scales of a trained layer's size, codes centred on zero."""
        c, f32 = self.case, self.case["dtype"] == "f32"
        lo, hi, mid = (1e-3, 2e-2, 8) if c["bits"] == 4 else (1e-4, 2e-3, 128)
        wq = torch.randint(-2 ** 31, 2 ** 31, (N, K * c["bits"] // 32), generator=self.gen, device="cuda", dtype=torch.int32)
        s = torch.rand((N, K // c["group"]), generator=self.gen, device="cuda").mul_(hi - lo).add_(lo).to(DTYPES[c["dtype"]][0])
        b = s * -mid
        if f32:
            b += self.normal(b.shape, torch.float32, 1e-3)
        return self.wrap(wq), self.wrap(s), self.wrap(b)

    def __del__(self):
        if self.graph is not None:
            self.ctx.graph_destroy(self.graph)
        for b in self.handles:
            b.free()


_context = None


def _ctx():
    """The process's one context, as a program has."""
    global _context
    if _context is None:
        _context = mlx_b200.Plugin().context(0)
    return _context


def prepare(case, seed):
    st = _State(case, _ctx(), seed)
    {"calls": _prepare_calls, "batch": _prepare_batch, "token": _prepare_token, "chain": _prepare_chain, "requant": _prepare_requant}[case["op"]](st)
    torch.cuda.synchronize()
    if case["op"] == "chain":  # run once (workspaces), then recorded
        _chain(st)
        st.ctx.sync()
        st.ctx.graph_begin()
        _chain(st)
        st.graph = st.ctx.graph_end()
    return st


def run(st):
    return {"calls": _run_calls, "batch": _run_batch, "token": _run_token, "chain": _run_chain, "requant": _run_requant}[st.case["op"]](st)


def _prepare_calls(st):
    c = st.case
    xt, yt = DTYPES[c["dtype"]][0], DTYPES[c["out"]][0]
    st.calls, st.out = [], []
    for _ in range(c["layers"]):
        x = st.wrap(st.normal((c["M"], c["K"]), xt))
        w, s, b = st.layer(c["N"], c["K"])
        t, y = st.empty((c["M"], c["N"]), yt)
        st.calls.append((x, w, s, b, y))
        st.out.append(t)


def _run_calls(st):
    c = st.case
    xd, yd = DTYPES[c["dtype"]][1], DTYPES[c["out"]][1]
    for x, w, s, b, y in st.calls:
        st.ctx.qmatmul(x, w, s, b, y, c["M"], c["K"], c["N"], c["bits"], c["group"], xd, xd, yd)
    return st.out


def _prepare_batch(st):
    c = st.case
    st.rows = _rows(c)
    st.x = [st.wrap(st.normal((m, c["K"]), torch.bfloat16)) for m in st.rows]
    st.w, st.s, st.b = zip(*(st.layer(c["N"], c["K"]) for _ in st.rows))
    st.out, st.y = zip(*(st.empty((m, c["N"]), DTYPES[c["out"]][0]) for m in st.rows))


def _run_batch(st):
    c = st.case
    st.ctx.qmatmul_batch(st.x, st.w, st.s, st.b, st.y, st.rows, c["K"], c["N"], c["bits"], c["group"], DTYPES[c["out"]][1])
    return list(st.out)


def _prepare_layers(st, widths):
    """Weights of every layer, and its buffers {name: (tensor, handle)}."""
    c = st.case
    st.x = st.wrap(st.normal((c["M"], c["K"]), torch.bfloat16))
    st.layers = []
    for _ in range(c["layers"]):
        st.layers.append(({n: (*st.layer(N, K), N, K) for n, N, K in _projections(c)},
                          {n: st.empty((c["M"], w), torch.bfloat16) for n, w in widths.items()}))


def _prepare_token(st):
    d, f = st.case["K"], st.case["N"]
    _prepare_layers(st, dict(r=d, q=d, k=d, v=d, o=d, r2=d, gate=f, up=f, down=d))


def _run_token(st):
    c, ctx, M = st.case, st.ctx, st.case["M"]

    def mm(name, src, dst):
        w, s, b, N, K = ws[name]
        ctx.qmatmul(src, w, s, b, dst, M, K, N, c["bits"], c["group"], BF16, BF16, BF16)

    h = st.x
    for ws, t in st.layers:
        r, r2 = t["r"][1], t["r2"][1]
        ctx.rms_norm(h, r, M, c["K"], EPS, BF16, BF16)
        for name in ("q", "k", "v"):
            mm(name, r, t[name][1])
        mm("o", t["q"][1], t["o"][1])
        ctx.rms_norm(t["o"][1], r2, M, c["K"], EPS, BF16, BF16)
        mm("gate", r2, t["gate"][1])
        mm("up", r2, t["up"][1])
        mm("down", t["gate"][1], t["down"][1])
        h = t["down"][1]
    return [{n: v[0] for n, v in t.items()} for _, t in st.layers]


def _prepare_chain(st):
    d, f = st.case["K"], st.case["N"]
    _prepare_layers(st, dict(qkv=3 * d, o=d, gateup=2 * f, m=f, d=d))
    st.out, st.h = st.empty((st.case["M"], d), torch.bfloat16)


def _chain(st):
    """a = q + k + v; o = Wo a; r = rms_norm(o); m = rms_norm(gate(r) * up(r)); d = Wd m; h = rms_norm(d)."""
    c, ctx, M, K = st.case, st.ctx, st.case["M"], st.case["K"]
    form = (c["bits"], c["group"])
    prev = None
    for ws, t in st.layers:
        (qkv, o, gateup, down), buf = (ws[n] for n in ("qkv", "o", "gateup", "down")), {n: v[1] for n, v in t.items()}
        if prev is None:
            ctx.qmatmul(st.x, *qkv[:3], buf["qkv"], M, K, 3 * K, *form, BF16, BF16, BF16)
        else:
            ctx.qmatmul_pro(prev, *qkv[:3], buf["qkv"], M, K, 3 * K, *form, BF16, PRO_RMS_NORM, K, EPS)
        ctx.qmatmul_pro(buf["qkv"], *o[:3], buf["o"], M, K, K, *form, BF16, PRO_SUM3, 3 * K, EPS)
        ctx.qmatmul_pro(buf["o"], *gateup[:3], buf["gateup"], M, K, gateup[3], *form, BF16, PRO_RMS_NORM, K, EPS)
        ctx.mul_rms_norm(buf["gateup"], buf["m"], M, c["N"], gateup[3], EPS)
        ctx.qmatmul(buf["m"], *down[:3], buf["d"], M, c["N"], K, *form, BF16, BF16, BF16)
        prev = buf["d"]
    ctx.rms_norm(prev, st.h, M, K, EPS, BF16, BF16)


def _run_chain(st):
    st.ctx.graph_launch(st.graph)
    return [st.out] + [v[0] for _, t in st.layers for v in t.values()]


def _prepare_requant(st):
    c = st.case
    N, K, t = c["N"], c["K"], DTYPES[c["dtype"]][0]
    st.src = st.wrap(st.normal((N, K), torch.float32, 0.02))
    packed, st.wq = st.empty((N, K * c["bits"] // 32), torch.int32)
    scales, st.sc = st.empty((N, K // c["group"]), t)
    biases, st.bi = st.empty((N, K // c["group"]), t)
    back, st.back = st.empty((N, K), t)
    st.out = [packed, scales, biases, back]


def _run_requant(st):
    c = st.case
    form, d = (c["N"], c["K"], c["bits"], c["group"]), DTYPES[c["dtype"]][1]
    st.ctx.quantize(st.src, st.wq, st.sc, st.bi, *form, d)
    st.ctx.dequantize(st.wq, st.sc, st.bi, st.back, *form, d, d)
    return st.out
