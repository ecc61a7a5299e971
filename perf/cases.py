"""Timed cases of the LLaMA/Qwen attention path and of the device-resident decoder around it, all through the
package's public entry points (``shainet_b200.attention``).

A case is one of six kinds of work a program hands to the package:

* ``host``      host arrays in, host array out, one blocking call per layer (``LlamaAttention.forward_cached``):
                the drop-in for a host program that keeps its activations on the CPU
* ``decode``    one new token per step through a stack of layers, device pointers (``forward_cached_dev``)
* ``batch``     one new token for each of several sequences of different lengths in lock step
                (``forward_batched_dev``)
* ``rows``      several new tokens of one sequence at once: a drafted continuation to verify, a short chat turn, a
                prompt, or a chunk of a prompt over what is cached already (``forward_cached_dev``)
* ``prompt``    a whole Q8_0 model over a prompt, logits and greedy token back on the host (``Decoder.run``)
* ``generate``  greedy tokens of a whole Q8_0 model over a filled cache (``Decoder.generate``)

Every pass starts from the same cache length (the rows of the pass before are dropped), so it can be repeated.
"""
import math
import random

import numpy as np
import torch

import shainet_b200 as S
from shainet_b200.attention import forward_batched_dev

# (query heads, kv heads, head_dim, RoPE theta, per-head q/k norm, projection biases)
HEADS = {
    "llama_1b": (32, 8, 64, 500000.0, False, False),
    "qwen3_8b": (32, 8, 128, 1e6, True, False),
    "qwen3_30b": (32, 4, 128, 1e6, True, False),
    "mha_16x64": (16, 16, 64, 10000.0, False, False),       # one query head per kv head
    "gqa_28x4": (28, 4, 128, 1e6, False, True),             # seven query heads per kv head, biased projections
    "mqa_32x2": (32, 2, 128, 1e6, False, False),            # sixteen query heads per kv head
}
TENSOR_ROWS = 64   # from this many new tokens on, attention is computed with TF32 operands


def listed():
    return [
        # The smallest call: a host program decoding one token of a short chat through four layers.
        dict(name="host_decode_short", kind="host", heads="llama_1b", layers=4, rows=1, ctx=700, kv="f32"),
        # One token through all layers of a 1B model in the middle of a 4k context: sixteen small dependent launches.
        dict(name="decode_4k", kind="decode", heads="llama_1b", layers=16, steps=2, ctx=4096, kv="f32"),
        # Long-context decode, the benchmarked head shape at 32k.
        dict(name="decode_32k", kind="decode", heads="qwen3_30b", layers=6, steps=3, ctx=32768, kv="f32"),
        # The same with the 16-bit cache at an odd length.
        dict(name="decode_bf16_12345", kind="decode", heads="qwen3_8b", layers=6, steps=3, ctx=12345, kv="bf16"),
        # A full server: 64 sequences of 1k to 32k positions in lock step.
        dict(name="batch_64_ragged", kind="batch", heads="qwen3_8b", layers=2, steps=1, batch=64, lo=1024, hi=32768,
             lengths=4001, kv="f32"),
        # A quiet server: eight chats of a few hundred to a few thousand positions.
        dict(name="batch_8_chats", kind="batch", heads="llama_1b", layers=8, steps=2, batch=8, lo=200, hi=4000,
             lengths=77, kv="f32"),
        # Verification of five drafted tokens over a 4k context.
        dict(name="verify_5", kind="rows", heads="qwen3_8b", layers=8, rows=5, ctx=4096, kv="f32"),
        # The next short user turn of a chat.
        dict(name="turn_40", kind="rows", heads="llama_1b", layers=16, rows=40, ctx=1900, kv="f32"),
        # The largest prompt: 8192 tokens of causal prefill.
        dict(name="prefill_8192", kind="rows", heads="qwen3_8b", layers=1, rows=8192, ctx=0, kv="f32"),
        # A ragged chunk of a long prompt over a 16-bit cache.
        dict(name="chunk_500_bf16", kind="rows", heads="llama_1b", layers=8, rows=500, ctx=3500, kv="bf16"),
        # Token generation of the 1B-shaped model, 16 layers, vocabulary 128256, over a 4k context.
        dict(name="generate_1b", kind="generate", heads="llama_1b", d_model=2048, ffn=8192, vocab=128256, layers=16,
             rows=1, ctx=4096, steps=16, kv="f32"),
        # The same model over a 4096-token prompt.
        dict(name="prompt_1b_4096", kind="prompt", heads="llama_1b", d_model=2048, ffn=8192, vocab=128256, layers=16,
             rows=4096, ctx=0, kv="f32"),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["host", "decode", "decode", "batch", "batch", "rows", "rows", "rows", "prompt", "prompt", "generate"])
    heads = rng.choice(["llama_1b", "llama_1b", "qwen3_8b", "qwen3_8b", "qwen3_30b", "mha_16x64", "gqa_28x4", "mqa_32x2"])
    kv = rng.choice(["f32", "f32", "bf16"])
    if kind == "host":
        return dict(kind=kind, heads=heads, layers=rng.randint(1, 4), rows=rng.choice([1, 1, _log(rng, 2, 512)]),
                    ctx=_log(rng, 16, 16384), kv=kv)
    if kind == "decode":
        return dict(kind=kind, heads=heads, layers=rng.randint(4, 8), steps=rng.randint(1, 4), ctx=_log(rng, 16, 32768), kv=kv)
    if kind == "batch":
        lo = _log(rng, 64, 2048)
        return dict(kind=kind, heads=heads, layers=rng.randint(1, 3), steps=rng.randint(1, 2), batch=_log(rng, 2, 64), lo=lo,
                    hi=lo * rng.randint(2, 8), lengths=rng.randint(1, 1 << 20), kv="f32" if heads == "gqa_28x4" else kv)
    if kind == "rows":
        rows = _log(rng, 2, 6000)
        ctx = rng.choice([0, _log(rng, 16, 16384)])
        return dict(kind=kind, heads=heads, layers=1 if rows > 1000 else rng.randint(2, 6), rows=rows, ctx=ctx, kv=kv)
    d_model = rng.choice([1024, 1536, 2048, 2048, 3072])
    model = dict(kind=kind, heads=heads, d_model=d_model, ffn=d_model * rng.choice([3, 4]), vocab=rng.choice([32000, 50257]),
                 layers=rng.randint(2, 4), kv=kv)
    if kind == "prompt":
        return dict(model, rows=_log(rng, 2, 1500), ctx=0)
    return dict(model, rows=rng.randint(1, 8), ctx=_log(rng, 16, 8192), steps=rng.randint(4, 12))


_ctx = None


def _context():
    """A program keeps one context for its device."""
    global _ctx
    if _ctx is None:
        _ctx = S.AttnContext(0)
    return _ctx


class Owned:
    """Library objects of one state, given back, newest first, when neither the state nor a tensor over their memory is
    left."""

    def __init__(self):
        self.objects = []

    def __del__(self):
        while self.objects:
            self.objects.pop().close()


class State:
    """What the program holds."""

    def __init__(self):
        self.owned = Owned()

    def own(self, obj):
        self.owned.objects.append(obj)
        return obj


class _DeviceArray:
    """fp32 device memory of the library, for torch, whose tensor keeps this object and with it the memory's owner."""

    def __init__(self, ptr, shape, owner):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": shape, "typestr": "<f4", "data": (ptr, False), "strides": None, "version": 3}


def _appended(st, cache, first, n):
    """The rows [first, first + n) of a cache's K and V, where they lie (fp32 caches: the library gives no pointers to
    16-bit rows)."""
    if cache.kv_format != "f32":
        return ()
    shape = (cache.num_kv_heads, cache.capacity, cache.head_dim)
    return tuple(torch.as_tensor(_DeviceArray(p, shape, st.owned), device="cuda")[:, first:first + n] for p in cache.device_ptrs())


def _attention(st, case, capacity, gen):
    H, KV, hd, theta, norm, bias = HEADS[case["heads"]]
    rnd = lambda n, sd, mean=0.0: (mean + sd * torch.randn(n, generator=gen)).numpy()
    kw = {}
    if norm:
        kw.update(q_norm=rnd(hd, 0.02, 1.0), k_norm=rnd(hd, 0.02, 1.0))
    if bias:
        kw.update(b_q=rnd(H * hd, 0.1), b_k=rnd(KV * hd, 0.1), b_v=rnd(KV * hd, 0.1))
    return st.own(S.LlamaAttention(_context(), H, KV, hd, theta, 1e-6, initial_capacity=capacity, kv_format=case["kv"], **kw))


def _lengths(case):
    r = random.Random(case["lengths"])
    return [_log(r, case["lo"], case["hi"]) for _ in range(case["batch"])]


def _normal(gen, *shape):
    return torch.randn(*shape, generator=gen, device="cuda")


def prepare(case, seed):
    st = State()
    cpu, gpu = torch.Generator().manual_seed(seed), torch.Generator("cuda").manual_seed(seed)
    H, KV, hd = HEADS[case["heads"]][:3]
    kind, layers = case["kind"], case["layers"]
    rows, ctx, steps = case.get("rows", 1), case.get("ctx", 0), case.get("steps", 1)
    st.kind, st.rows, st.ctx, st.steps = kind, rows, ctx, steps
    if kind in ("prompt", "generate"):
        _prepare_model(st, case, seed, cpu, gpu)
    elif kind == "batch":
        st.lens = _lengths(case)
        st.layers = []
        for l in range(layers):
            attns = [_attention(st, case, n + steps, cpu.manual_seed(seed + l)) for n in st.lens]
            for b, (a, n) in enumerate(zip(attns, st.lens)):
                a.cache.fill_normal(n, seed + 1000 * l + b)
            st.layers.append([a.cache for a in attns])
        st.scale = 1.0 / math.sqrt(hd)
        B = len(st.lens)
        st.q, st.k, st.v = (_normal(gpu, steps, layers, B, n * hd) for n in (H, KV, KV))
        st.out = torch.empty_like(st.q)
        st.ptrs = [[[t[s, l].data_ptr() for t in (st.q, st.k, st.v, st.out)] for l in range(layers)] for s in range(steps)]
        # at most thirty caches' new rows are handed back beside the outputs
        st.new = [_appended(st, c, n, steps) for cs in st.layers for c, n in zip(cs, st.lens)][:30]
    else:
        st.layers = [_attention(st, case, ctx + rows * steps, cpu) for _ in range(layers)]
        for l, a in enumerate(st.layers):
            a.cache.fill_normal(ctx, seed + 1000 * l)
        st.q, st.k, st.v = (_normal(gpu, steps, layers, rows, n * hd) for n in (H, KV, KV))
        if kind == "host":
            st.q, st.k, st.v = (t[0].cpu().numpy() for t in (st.q, st.k, st.v))
        else:
            st.out = torch.empty_like(st.q)
            st.ptrs = [[[t[s, l].data_ptr() for t in (st.q, st.k, st.v, st.out)] for l in range(layers)] for s in range(steps)]
        st.new = [_appended(st, a.cache, ctx, rows * steps) for a in st.layers]
    torch.cuda.synchronize()
    return st


def _prepare_model(st, case, seed, cpu, gpu):
    """Weights N(0, 0.02) as Q8_0: int8 values and one scale per 32 inputs, on the device; embedding and norms on the host."""
    H, KV, hd = HEADS[case["heads"]][:3]
    d, ffn, vocab = case["d_model"], case["ffn"], case["vocab"]
    st.weights = []

    def weight(K, N):
        q = _normal(gpu, N, K).mul_(32.0).round_().clamp_(-127, 127).to(torch.int8)
        s = (0.02 / 32.0) * (0.8 + 0.4 * torch.rand(N, (K + 31) // 32, generator=gpu, device="cuda"))
        st.weights.append((q, s))
        torch.cuda.synchronize()   # the library works on a stream of its own
        return st.own(S.Q8Weight.wrap(_context(), q.data_ptr(), s.data_ptr(), K, N))

    gain = lambda: (1.0 + 0.05 * torch.randn(d, generator=cpu)).numpy()
    blocks, st.attns = [], []
    for l in range(case["layers"]):
        a = _attention(st, case, st.ctx + st.rows + st.steps + 1, cpu)
        a.cache.fill_normal(st.ctx, seed + 1000 * l)
        st.attns.append(a)
        blocks.append(st.own(S.LlamaBlock(_context(), a, d, 1e-5, gain(), weight(d, H * hd), weight(d, KV * hd), weight(d, KV * hd),
                                          weight(H * hd, d), gain(), weight(d, ffn), weight(d, ffn), weight(ffn, d))))
    embedding = _normal(gpu, vocab, d).mul_(0.5).cpu().numpy()
    st.decoder = st.own(S.Decoder(_context(), blocks, embedding, gain(), weight(d, vocab), None, 1e-5))
    st.ids = np.asarray(torch.randint(0, vocab, (st.rows,), generator=cpu), np.int32)
    st.new = [_appended(st, a.cache, st.ctx, st.rows + st.steps - 1) for a in st.attns]


def run(st):
    if st.kind == "prompt":
        for a in st.attns:
            a.cache.truncate(st.ctx)
        return st.decoder.run(st.ids), st.new
    if st.kind == "generate":
        for a in st.attns:
            a.cache.truncate(st.ctx)
        return st.decoder.generate(st.ids, st.steps), st.new
    if st.kind == "batch":
        for caches in st.layers:
            for c, n in zip(caches, st.lens):
                c.truncate(n)
        for s in range(st.steps):
            for caches, (q, k, v, out) in zip(st.layers, st.ptrs[s]):
                forward_batched_dev(_context(), caches, q, k, v, out, st.scale)
        return st.out, st.new
    for a in st.layers:
        a.cache.truncate(st.ctx)
    if st.kind == "host":
        return [a.forward_cached(st.q[l], st.k[l], st.v[l]) for l, a in enumerate(st.layers)], st.new
    for s in range(st.steps):
        for a, (q, k, v, out) in zip(st.layers, st.ptrs[s]):
            a.forward_cached_dev(q, k, v, out, st.rows)
    return st.out, st.new


def work(case):
    H, KV, hd = HEADS[case["heads"]][:3]
    es = 2 if case["kv"] == "bf16" else 4
    rows, steps, layers = case.get("rows", 1), case.get("steps", 1), case["layers"]
    nbytes = flops = 0

    def attention(ctx, T, ends=True):
        """Cached rows read, new rows read and written, q read and the output written; every visible pair two products.
        ends=False: q, the new rows and the output stay inside a model."""
        nonlocal nbytes, flops
        nbytes += 2 * KV * hd * es * (ctx + T)
        if ends:
            nbytes += 4 * T * hd * (2 * H + 2 * KV)
        flops += 4 * hd * H * (T * ctx + T * (T + 1) // 2)

    if case["kind"] == "batch":
        for n in _lengths(case):
            for s in range(steps):
                attention(n + s, 1)
        return {"bytes": nbytes * layers, "flops": flops * layers}
    if case["kind"] in ("host", "decode", "rows"):
        for s in range(steps):
            attention(case["ctx"] + rows * s, rows)
        return {"bytes": nbytes * layers, "flops": flops * layers}
    d, ffn, vocab = case["d_model"], case["ffn"], case["vocab"]
    per_layer = d * (H + 2 * KV) * hd + H * hd * d + 3 * d * ffn
    head = d * vocab
    weight_bytes = lambda n: n + 4 * (n // 32)
    passes = [rows] + [1] * (steps - 1)   # the prompt, then single tokens
    at, total_b, total_f = case["ctx"], 0, 0
    for T in passes:
        nbytes = flops = 0
        attention(at, T, ends=False)
        total_b += layers * (nbytes + weight_bytes(per_layer)) + weight_bytes(head) + 4 * T * d
        total_f += layers * (flops + 2 * T * per_layer) + 2 * head
        at += T
    return {"bytes": total_b, "flops": total_f}


def tolerance(case):
    """fp32 arithmetic: sums in another order.  From TENSOR_ROWS new tokens on the operands of attention carry TF32's ten
    mantissa bits.  With a 16-bit cache a new row's element that lies at a rounding boundary may go either way.  A model
    compounds its layers."""
    model = case["kind"] in ("prompt", "generate")
    if case.get("rows", 1) >= TENSOR_ROWS:
        return {"rel": 2e-3 if model else 1e-3}
    if case["kv"] == "bf16":
        return {"rel": 1e-3 if model else 1e-4}
    return {"rel": 1e-4 if model else 1e-5}
