"""The work a user of this framework has it do, as cases that can be timed and compared.

A case is a dict of plain values.  `listed()` gives the fixed ones, `draw(rng)` one more of the same ranges,
`prepare(case, seed)` what a program has in hand before the call, `run(state)` one pass through the public entry points,
`work(case)` the bytes and operations of a pass and `tolerance(case)` how far two correct implementations may be apart.

Kinds of work:
  gemv     one activation row through one packed matrix, the single call a host program issues by itself
  matmul   a block of activation rows through one packed matrix (`GpuWeight::matmul_x`)
  decode   one token of one sequence through the whole captured stack, input row in and hidden row out
  batch    one token of each of several independent sequences of different lengths through the whole captured stack
  prefill  the positions of a prompt (or of the next chunk of one) through the whole stack
  load     quantisation of one f32 matrix into the packed 4-bit format at model load

Model shapes are those of nve_b200.bench_random.SHAPES.  A program loads a model once and serves many inputs with it:
weights, caches and the recorded graph of a stack are kept from one `prepare` of a case to the next (one stack at a
time, the library holds one recorded graph), the inputs are made from the seed.
"""
import math

import torch

from nve_b200 import cuda_kernels as ck
from nve_b200.bench_random import SHAPES, build_state, decode_bytes_per_token, layer_weight_bytes, make_w4, w4_bytes
from nve_b200.decode_graph import CapturedSequence, StaticDecodeGraph
from nve_b200.gpu_layer import (BatchedDecodeScratch, BatchedKvCache, RoutingConfig, gpu_layer_forward_decode_batch,
                                gpu_layer_forward_prefill, matmul_x)

MODEL_SEED = 20
DTYPES = {"f16": torch.float16, "bf16": torch.bfloat16}


def listed():
    return [
        # the smallest call: the up projection of a 1B model for one token, weights on the 16-bit activation route
        dict(name="gemv_1b_up", kind="gemv", n=8192, k=2048, route="w4a16"),
        # a handful of rows through one wide-K projection with bf16 activations: draft verification, a short prompt tail
        dict(name="matmul_8b_down_bf16_20", kind="matmul", m=20, n=4096, k=14336, dtype="bf16"),
        # chat with a small model early in the conversation: short kernels, launches count
        dict(name="decode_1b_ctx256", kind="decode", model="1b", context=256, route="mixed", awq=False),
        # the headline: 8B model, half of the layers on int8 activations
        dict(name="decode_8b_ctx1024", kind="decode", model="8b", context=1024, route="mixed", awq=False),
        # long document, AWQ checkpoint: activation multipliers and 16-bit activations in every layer
        dict(name="decode_8b_ctx16384_awq", kind="decode", model="8b", context=16384, route="w4a16", awq=True),
        # the largest model that one GPU serves: bound by the 43 GB of weights
        dict(name="decode_70b_ctx1024", kind="decode", model="70b", context=1024, route="mixed", awq=False),
        # a few users on a mid-size model (three query heads per KV head), sequences of different lengths
        dict(name="batch_3b_7_ctx2000", kind="batch", model="3b", batch=7, context=2000),
        # a full serving batch
        dict(name="batch_8b_64_ctx1024", kind="batch", model="8b", batch=64, context=1024),
        # a short question
        dict(name="prefill_8b_61", kind="prefill", model="8b", rows=61, start=0),
        # a page of text as the next chunk of a conversation
        dict(name="prefill_3b_300_at_700", kind="prefill", model="3b", rows=300, start=700),
        # a long prompt, not a multiple of any tile
        dict(name="prefill_8b_1777", kind="prefill", model="8b", rows=1777, start=0),
        # loading: the gate projection of an 8B model, f32 in, packed out
        dict(name="load_8b_gate", kind="load", n=14336, k=4096, awq=False),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["gemv", "matmul", "decode", "decode", "batch", "batch", "prefill", "prefill", "load"])
    if kind == "gemv":  # any number of rows; K in whole quantisation blocks
        return dict(kind=kind, n=_log(rng, 256, 32768), k=32 * _log(rng, 16, 512), route=rng.choice(["w4a16", "w4a8"]))
    if kind == "matmul":  # the GEMM takes K in multiples of 64
        return dict(kind=kind, m=_log(rng, 2, 128), n=_log(rng, 512, 16384), k=64 * _log(rng, 16, 224),
                    dtype=rng.choice(["f16", "bf16"]))
    if kind == "decode":
        awq = rng.random() < 0.3
        return dict(kind=kind, model=rng.choice(["1b", "3b", "8b"]), context=_log(rng, 16, 16384),
                    route="w4a16" if awq else rng.choice(["mixed", "w4a8", "w4a16"]), awq=awq)
    if kind == "batch":
        b = _log(rng, 2, 64)
        return dict(kind=kind, model=rng.choice(["1b", "3b", "8b"]), batch=b, context=_log(rng, 32, min(8192, 65536 // b)))
    if kind == "prefill":
        rows = _log(rng, 2, 1777)
        most = max(1, min(3000, 1777 * 1777 // (2 * rows) - rows // 2))  # no more attention work than the largest listed
        return dict(kind=kind, model=rng.choice(["1b", "3b", "8b"]), rows=rows, start=rng.choice([0, rng.randrange(most)]))
    return dict(kind=kind, n=_log(rng, 512, 14336), k=32 * _log(rng, 32, 448), awq=rng.random() < 0.5)


# ------------------------------------------------------------------------------------------------ stacks
_stack = {"key": None, "value": None}


def _drop_stack():
    old = _stack["value"]
    _stack.update(key=None, value=None)
    if old is not None:
        torch.cuda.synchronize()
        if "graph" in old:
            old["graph"].destroy()
        old.clear()
        torch.cuda.empty_cache()


def _caches(layers, shape, stream_id):
    """One tensor for all layers' K (or V) rows, filled ~N(0, 1); the caches of the layers are views of it."""
    t = torch.empty((layers,) + shape, dtype=torch.float16, device="cuda")
    for li in range(layers):
        ck.fill_normal(t[li].numel(), MODEL_SEED, stream_id + 2 * li, dtype=torch.float16, out=t[li].view(-1))
    return t


def _multiplier(k, gen):
    """AWQ multipliers as calibration leaves them: around 1, within a factor of two."""
    return torch.exp2(torch.rand(k, generator=gen) * 2 - 1).cuda()


def _build_stack(case):
    shape = SHAPES[case["model"]]
    kind, layers = case["kind"], shape.num_layers
    max_seq = case["rows"] + case["start"] if kind == "prefill" else case["context"]
    state, importance = build_state(shape, MODEL_SEED, max_seq if kind != "batch" else 1, max_seq=max_seq, fill_kv=False)
    if case.get("route") == "w4a16":
        state.routing = RoutingConfig(no_w4a8=True)
    elif case.get("route") == "w4a8":
        state.routing = RoutingConfig(threshold=2.0)
    if case.get("awq"):
        gen = torch.Generator().manual_seed(MODEL_SEED)
        for w in state.layer_weights:
            qkv, gate_up = _multiplier(w.q_proj.k, gen), _multiplier(w.gate_proj.k, gen)
            w.q_proj.awq_scales = w.k_proj.awq_scales = w.v_proj.awq_scales = qkv
            w.gate_proj.awq_scales = w.up_proj.awq_scales = gate_up
            w.o_proj.awq_scales, w.down_proj.awq_scales = _multiplier(w.o_proj.k, gen), _multiplier(w.down_proj.k, gen)
    # norm weights well below one, as trained checkpoints have them: a layer adds a small part to the residual stream
    gen = torch.Generator().manual_seed(MODEL_SEED + 1)
    norm = min(0.3, 1200 / shape.hidden)
    for w in state.layer_weights:
        w.input_norm, w.post_attn_norm = (
            (norm * (1 + torch.randn(shape.hidden, generator=gen) / 6)).half().cuda() for _ in range(2))
    rows = (shape.num_kv_heads, max_seq, shape.head_dim)
    if kind == "batch":
        rows = (case["batch"],) + rows
    k, v = _caches(layers, rows, 500000), _caches(layers, rows, 500001)
    held = dict(state=state, k=k, v=v, layers=layers)
    if kind == "batch":
        kv = BatchedKvCache(list(k.unbind(0)), list(v.unbind(0)), case["batch"], max_seq)
        b = case["batch"]
        # sequences of different ages: from a quarter of the longest on
        lens = [max(1, max_seq - (3 * max_seq // 4) * i // max(1, b - 1)) for i in range(b)]
        d_len = torch.tensor(lens, dtype=torch.int32, device="cuda")
        d_pos = d_len - 1
        x = torch.zeros((b, shape.hidden), dtype=torch.float16, device="cuda")
        scratch = BatchedDecodeScratch.make(state, b, shape.hidden, shape.ffn)

        def record(_pos, _len):
            h, res = x, None
            for li in range(layers):  # the add at the end of a layer rides on the next layer's first launch
                r = gpu_layer_forward_decode_batch(h, li, state, kv, d_pos, d_len, scratch, residual=res, defer_add=li < layers - 1)
                h, res = r if li < layers - 1 else (r, None)
            held["out"] = h

        held.update(kv=kv, x=x, lens=(d_pos, d_len), scratch=scratch, graph=CapturedSequence(record))
        return held
    state.kv_cache.k, state.kv_cache.v = list(k.unbind(0)), list(v.unbind(0))
    if kind == "decode":
        held["graph"] = StaticDecodeGraph(state, shape.hidden, shape.ffn, importance)
        held["graph"].capture()
    return held


def _the_stack(case):
    key = tuple(sorted((k, v) for k, v in case.items() if k != "name"))
    if _stack["key"] != key:
        _drop_stack()
        _stack.update(value=_build_stack(case), key=key)
        torch.cuda.synchronize()
    return _stack["value"]


# ------------------------------------------------------------------------------------------------ the five functions
def prepare(case, seed):
    ck.set_pdl(True)  # as a decoding program switches it on: kernels may start while their predecessor drains
    kind = case["kind"]
    if kind in ("gemv", "matmul"):
        dt = DTYPES[case.get("dtype", "f16")]
        m, n, k = case.get("m", 1), case["n"], case["k"]
        return dict(kind=kind, route=case.get("route"), w=make_w4(n, k, seed, 1),
                    x=ck.fill_normal(m * k, seed, 2, dtype=dt).view(m, k))
    if kind == "load":
        n, k = case["n"], case["k"]
        awq = torch.exp2(torch.rand(k, generator=torch.Generator("cuda").manual_seed(seed), device="cuda") * 2 - 1) \
            if case["awq"] else None
        return dict(kind=kind, w=ck.fill_normal(n * k, seed, 1, scale=0.02).view(n, k), awq=awq)
    hidden = SHAPES[case["model"]].hidden
    rows = {"decode": 1, "batch": case.get("batch"), "prefill": case.get("rows")}[kind]
    x = ck.fill_normal(rows * hidden, seed, 42, dtype=torch.float16).view(rows, hidden)
    return dict(kind=kind, x=x, stack=_the_stack(case), pos=case.get("start", case.get("context", 1) - 1))


def run(state):
    kind, x = state["kind"], state.get("x")
    if kind == "gemv":
        w = state["w"]
        if state["route"] == "w4a16":
            return ck.fused_matvec_w4a16(x, w.nibbles, w.scales, None, w.n, w.k)
        xq, xs = ck.quantize_f16_q8(x)
        return xq, xs, ck.matvec_w4a8(xq, xs, w.nibbles, w.scales, w.n, w.k)
    if kind == "matmul":
        return matmul_x(x, state["w"])
    if kind == "load":
        return ck.q4_quantize(state["w"], state["awq"])
    s = state["stack"]
    if kind == "decode":
        h = s["graph"].replay(x, state["pos"])
    elif kind == "batch":
        ck.device_copy(s["x"], x)
        s["graph"].replay(0, 1)  # positions travel in the sequences' own device arrays
        h = s["out"].clone()
    else:
        h = x
        for li in range(s["layers"]):
            h = gpu_layer_forward_prefill(h, li, s["state"], state["pos"])
    return dict(hidden=h, k=s["k"], v=s["v"])


def work(case):
    kind = case["kind"]
    if kind in ("gemv", "matmul"):
        m, n, k = case.get("m", 1), case["n"], case["k"]
        codes = k + k // 8 if case.get("route") == "w4a8" else 0
        return {"bytes": w4_bytes(n, k) + 2 * m * (n + k) + codes, "flops": 2 * m * n * k}
    if kind == "load":
        n, k = case["n"], case["k"]
        return {"bytes": 4 * n * k + w4_bytes(n, k) + (4 * k if case["awq"] else 0), "flops": 3 * n * k}
    s = SHAPES[case["model"]]
    params = s.num_layers * layer_weight_bytes(s) * 8 // 5  # 0.625 bytes per weight
    row = 2 * s.num_kv_heads * s.head_dim * 2  # K and V of one position, 16 bit
    att = 4 * s.num_heads * s.head_dim         # operations per (query row, position)
    if kind == "decode":
        return {"bytes": decode_bytes_per_token(s, case["context"]) + 4 * s.hidden,
                "flops": 2 * params + s.num_layers * att * case["context"]}
    if kind == "batch":
        b, c = case["batch"], case["context"]
        seen = sum(max(1, c - (3 * c // 4) * i // max(1, b - 1)) for i in range(b))
        return {"bytes": s.num_layers * (layer_weight_bytes(s) + row * seen) + 4 * b * s.hidden,
                "flops": 2 * b * params + s.num_layers * att * seen}
    r, at = case["rows"], case["start"]
    pairs = r * at + r * (r + 1) // 2
    return {"bytes": s.num_layers * (layer_weight_bytes(s) + row * (at + r)) + 4 * r * s.hidden,
            "flops": 2 * r * params + s.num_layers * att * pairs}


def tolerance(case):
    kind = case["kind"]
    if kind == "load":
        return "exact"
    if kind == "gemv":  # one f16 rounding of an f32 sum; int8 codes are whole numbers and stay the same
        return {"rel": 1e-3, "max": 1e-2, "differ": 0.0}
    if kind == "matmul":
        return {"rel": 1e-2 if case["dtype"] == "bf16" else 2e-3}
    # f16 hidden state through every layer of a stack; where layers run on int8 activations, one code that rounds the
    # other way is an error of a 1/127th of its group's largest value for every layer behind it
    return {"rel": 2e-2 if case.get("route") in ("mixed", "w4a8") else 1e-2}
