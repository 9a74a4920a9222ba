"""Performance cases of the dequantize-fused linear path: what a program built on this package has it do, through the
package's public entry points.

A case is a dict of plain values with a ``kind``:

* ``linear``     one quantised linear: ``DequantDot`` (``front`` "node") or a ``jit``-prepared ``QuantLinear`` module
                 (``front`` "module"), from one row (decode) to thousands (prefill);
* ``mlp``        a SwiGLU MLP, gate / up / down, as ``ShardedMLP`` on one GPU, with or without the RMSNorm prologue;
* ``layer``      one decoder layer for one new token, ``DecoderLayer``;
* ``attention``  one decoding step of an attention layer, ``DecodeAttention``.

``graph`` marks programs that capture their decode step once and replay it, as serving loops do; the others issue
every call from Python.  Weights are random in the package's formats (uint4 packed two per byte, or uint8, with
group-wise or per-row scales and zero-points), activations and caches ~N(0, 1).
"""
from __future__ import annotations

import math

import torch

from nnfusion_b200.attention import DecodeAttention
from nnfusion_b200.decoder_layer import DecoderLayer
from nnfusion_b200.jit import QuantLinear, jit
from nnfusion_b200.linear import DequantDot, DeviceWeight
from nnfusion_b200.tp import ShardedMLP

_DT = {"f16": torch.float16, "f32": torch.float32}


def _linear(name, M, N, K, *, bits=4, group=128, dtype="f16", norm=False, epilogue="none", front="node", graph=False):
    """group 0: one scale and zero-point per weight row."""
    c = dict(kind="linear", M=M, N=N, K=K, bits=bits, group=group, dtype=dtype, norm=norm, epilogue=epilogue,
             front=front, graph=graph)
    return dict(c, name=name) if name else c


def _mlp(name, M, hidden, inter, *, norm=True, graph=False):
    c = dict(kind="mlp", M=M, hidden=hidden, inter=inter, norm=norm, graph=graph)
    return dict(c, name=name) if name else c


def _layer(name, heads, kv_heads, inter, position):
    c = dict(kind="layer", heads=heads, kv_heads=kv_heads, inter=inter, position=position)
    return dict(c, name=name) if name else c


def _attention(name, heads, kv_heads, position):
    c = dict(kind="attention", heads=heads, kv_heads=kv_heads, position=position)
    return dict(c, name=name) if name else c


def listed():
    return [
        # the smallest call: a narrow projection with bias of a torch module, one token; latency of a call
        _linear("module_m1_1024x4096_bias", 1, 1024, 4096, epilogue="bias", front="module"),
        # single-token decode, 7B-shaped up projection (the benchmark's headline shape), one Python call per linear
        _linear("decode_m1_11008x4096", 1, 11008, 4096),
        # a few sequences decoded together (an odd number), 7B-shaped down projection with the residual added
        _linear("decode_m5_4096x11008_add", 5, 4096, 11008, epilogue="add"),
        # the reference's own CPU-runnable graph: fp32 activations, uint8 weights with one scale per row, 16 rows
        _linear("u8_f32_m16_4096x4096", 16, 4096, 4096, bits=8, group=0, dtype="f32"),
        # single-token decode of a 70B-shaped MLP replayed from a graph: the largest memory-bound step
        _mlp("mlp70b_m1_graph", 1, 8192, 28672, norm=False, graph=True),
        # 16 sequences decoded together through a 7B-shaped MLP
        _mlp("mlp7b_m16", 16, 4096, 11008),
        # a decoder layer generating one token behind 2048 cached ones
        _layer("layer7b_pos2048", 32, 32, 11008, 2048),
        # a decoding step with grouped queries behind a long context
        _attention("attention_64q8kv_pos8191", 64, 8, 8191),
        # between decode and prefill: a large decode batch, or the prompt of a short request
        _linear("batch_m48_4096x11008", 48, 4096, 11008),
        # a prompt of ordinary, ragged length through a 7B-shaped MLP
        _mlp("mlp7b_m333", 333, 4096, 11008),
        # a long prompt, 7B-shaped up projection: the largest compute-bound call
        _linear("prefill_m4096_11008x4096", 4096, 11008, 4096),
        # the fp32 / uint8 format with a batch, ragged row count, bias
        _linear("u8_f32_m1000_4096x4096_bias", 1000, 4096, 4096, bits=8, group=0, dtype="f32", epilogue="bias"),
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _dim(rng, lo, hi, step):
    return max(lo, _log_uniform(rng, lo, hi) // step * step)


def _cost(case):
    w = work(case)
    return w["bytes"] / 6.5e12 + w["flops"] / 1.6e15


def draw(rng):
    most = 0.9 * max(_cost(c) for c in listed() if c["kind"] == "linear")  # the long prompt: no drawn case costs more
    while True:
        u = rng.random()
        if u < 0.55:
            bits = 8 if rng.random() < 0.25 else 4
            dtype = "f32" if rng.random() < (0.6 if bits == 8 else 0.1) else "f16"
            group = rng.choice([0, 0, 128, 64]) if bits == 8 else rng.choice([128, 128, 128, 128, 256, 0])
            M = _log_uniform(rng, 1, 4096)
            N = _dim(rng, 256, 28672, 16)
            if rng.random() < 0.3:
                N += rng.randrange(1, 16)  # not a whole number of tiles
            K = _dim(rng, 512, 28672, max(group, 128))
            epilogue = rng.choice(["none", "none", "bias", "add", "silu_mul"])
            norm = rng.random() < 0.3
            front = "module" if not norm and epilogue in ("none", "bias") and dtype == "f16" and rng.random() < 0.3 else "node"
            case = _linear(None, M, N, K, bits=bits, group=group, dtype=dtype, norm=norm, epilogue=epilogue, front=front,
                           graph=M <= 16 and rng.random() < 0.3)
        elif u < 0.75:
            M = _log_uniform(rng, 1, 2048)
            case = _mlp(None, M, _dim(rng, 1024, 8192, 128), _dim(rng, 2048, 28672, 128), norm=rng.random() < 0.7,
                        graph=M <= 16 and rng.random() < 0.5)
        elif u < 0.85:
            heads = rng.choice([16, 24, 32, 40, 64])
            case = _layer(None, heads, heads // rng.choice([1, 1, 4, 8]), _dim(rng, 4096, 28672, 128),
                          _log_uniform(rng, 16, 8191))
        else:
            heads = rng.choice([8, 16, 32, 40, 64])
            case = _attention(None, heads, heads // rng.choice([1, 2, 4, 8]), _log_uniform(rng, 16, 16383))
        if _cost(case) <= most and 6 * work(case)["bytes"] < 8e9:
            return case


# ---------------------------------------------------------------------------------------------------- inputs


class _Inputs:
    """Seeded tensors on the GPU."""

    def __init__(self, seed):
        self.gen = torch.Generator(device="cuda")
        self.gen.manual_seed(seed)

    def normal(self, *shape, dtype=torch.float16):
        return torch.randn(*shape, device="cuda", generator=self.gen).to(dtype)

    def uniform(self, lo, hi, *shape):
        return torch.rand(*shape, device="cuda", generator=self.gen) * (hi - lo) + lo

    def bytes(self, lo, hi, *shape):
        return torch.randint(lo, hi, shape, dtype=torch.uint8, device="cuda", generator=self.gen)

    def weight(self, N, K, bits=4, group=128, scale_dtype=torch.float16):
        group = group or K
        G = K // group
        if bits == 4:
            wq, zp = self.bytes(0, 256, N, K // 2), self.bytes(0, 256, N, (G + 1) // 2)
            scale = self.uniform(0.002, 0.02, N, G)
        else:
            wq, zp = self.bytes(0, 256, N, K), self.bytes(120, 137, N, G)
            scale = self.uniform(0.001, 0.01, N, G)
        return DeviceWeight(N, K, bits, group, wq, scale.to(scale_dtype), zp)


def _captured(step):
    """The step captured as a CUDA graph (run once before: first-call set-up and workspaces stay outside)."""
    step()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = step()

    def replay():
        graph.replay()
        return out
    return replay


def prepare(case, seed):
    r = _Inputs(seed)
    kind = case["kind"]
    if kind == "linear":
        M, N, K, dt = case["M"], case["N"], case["K"], _DT[case["dtype"]]
        dual = case["epilogue"] == "silu_mul"
        w, w2 = (r.weight(N, K, case["bits"], case["group"], dt) if i == 0 or dual else None for i in range(2))
        bias = r.uniform(-1, 1, N) if case["epilogue"] == "bias" else None
        x = r.normal(M, K, dtype=dt)
        if case["front"] == "module":
            m = QuantLinear(K, N, case["bits"], w.group, bias is not None, dt).cuda()
            for name, t in (("wq", w.wq), ("scale", w.scale), ("zp", w.zp)):
                getattr(m, name).copy_(t)
            if bias is not None:
                m.bias.data.copy_(bias)
            m = jit(m)
            x = x.view(1, M, K)  # [batch, tokens, features]

            def step():
                return m(x)
        else:
            node = DequantDot(w, w2, gain=r.uniform(0.9, 1.1, K) if case["norm"] else None, bias=bias,
                              add=case["epilogue"] == "add")
            if case["epilogue"] == "add":
                addend = r.normal(M, N, dtype=dt)

                def step():
                    return node(x, addend=addend)
            else:
                def step():
                    return node(x)
    elif kind == "mlp":
        H, I = case["hidden"], case["inter"]
        gate, up, down = r.weight(I, H), r.weight(I, H), r.weight(H, I)
        mlp = ShardedMLP(gate, up, down, gain=r.uniform(0.9, 1.1, H) if case["norm"] else None)
        x = r.normal(case["M"], H)

        def step():
            return mlp(x)
    elif kind == "layer":
        heads, kv, pos = case["heads"], case["kv_heads"], case["position"]
        H, I = 128 * heads, case["inter"]
        shapes = ((H, H), (128 * kv, H), (128 * kv, H), (H, H), (I, H), (I, H), (H, I))
        layer = DecoderLayer(*(r.weight(n, k) for n, k in shapes), r.uniform(0.9, 1.1, H), r.uniform(0.9, 1.1, H),
                             heads=heads, kv_heads=kv, capacity=(pos + 256) // 256 * 256)
        for cache in (layer.attn.k_cache, layer.attn.v_cache):
            cache.copy_(r.normal(*cache.shape))
        x = r.normal(1, H)

        def step():
            return layer(x, pos), layer.attn.k_cache, layer.attn.v_cache
    else:
        heads, kv, pos = case["heads"], case["kv_heads"], case["position"]
        node = DecodeAttention(heads, kv, 128, (pos + 256) // 256 * 256, "cuda")
        for cache in (node.k_cache, node.v_cache):
            cache.copy_(r.normal(*cache.shape))
        q, k, v = r.normal(heads * 128), r.normal(kv * 128), r.normal(kv * 128)

        def step():
            return node(q, k, v, pos), node.k_cache, node.v_cache
    return _captured(step) if case.get("graph") else step


def run(state):
    return state()


# ---------------------------------------------------------------------------------------------------- what a pass costs


def _weight_bytes(N, K, bits=4, group=128, scale_bytes=2):
    G = K // (group or K)
    return N * (K * bits // 8 + G * scale_bytes + ((G + 1) // 2 if bits == 4 else G))


def work(case):
    kind = case["kind"]
    if kind == "linear":
        M, N, K, e = case["M"], case["N"], case["K"], _DT[case["dtype"]].itemsize
        sets = 2 if case["epilogue"] == "silu_mul" else 1
        b = sets * _weight_bytes(N, K, case["bits"], case["group"], e) + e * M * (K + N)
        b += 4 * K if case["norm"] else 0
        b += {"bias": 4 * N, "add": e * M * N}.get(case["epilogue"], 0)
        return {"bytes": b, "flops": 2 * sets * M * N * K}
    if kind == "mlp":
        M, H, I = case["M"], case["hidden"], case["inter"]
        b = 2 * _weight_bytes(I, H) + _weight_bytes(H, I) + 2 * 2 * M * H + (4 * H if case["norm"] else 0)
        return {"bytes": b, "flops": 6 * M * H * I}
    heads, kv, rows = case["heads"], case["kv_heads"], case["position"] + 1
    attn = {"bytes": 2 * 128 * (2 * kv * rows + 2 * heads + 2 * kv), "flops": 4 * 128 * heads * rows}
    if kind == "attention":
        return attn
    H, I, Q = 128 * heads, case["inter"], 128 * (heads + 2 * kv)
    b = _weight_bytes(Q, H) + _weight_bytes(H, H) + 2 * _weight_bytes(I, H) + _weight_bytes(H, I)
    b += 2 * 128 * 2 * kv * rows + 2 * 4 * H + 2 * 2 * H
    return {"bytes": b, "flops": 2 * H * (Q + H + 3 * I) + attn["flops"]}


def tolerance(case):
    kind = case["kind"]
    if kind == "linear":
        if case["dtype"] == "f32" and case["M"] <= 16 and (case["bits"] == 8 or case["M"] <= 8):
            return {"rel": 2e-5}  # fp32 activations as two fp16 halves (22 bits), fp32 sums
        return {"rel": 1e-3}      # fp16 operands (11 bits) for the tensor cores, fp32 sums
    if kind == "attention":
        return {"rel": 1e-3}      # fp16 in and out, fp32 in between
    return {"rel": 3e-3}          # two to five such steps in a row, fp16 between them
