"""The calls that a user of this library makes, from one decoded token to a long prompt, as cases that can be timed.

An inference engine calls the library once per layer and step: the MoE block of a token, of a decode batch or of a prompt
chunk, on device or on host buffers; the whole stack of layers; the experts alone with a selection of its own; the block
inside a hyper-connection layer; the GEMV of a single quantised matrix.  A pass is one such step through a few layers
(through one layer where the call is long), each layer with its own weights and its own input, so that the weights of a
pass come from HBM as they do in a model of dozens of layers, and no layer's rounding reaches the next one's routing.

    listed()  the cases            draw(rng)  one more of the same ranges
    prepare(case, seed)            weights, inputs and output buffers, as a program keeps them
    run(state)                     one pass; returns its outputs
    work(case), tolerance(case)    what a pass cannot do without; how far another implementation may be off
"""
import math

import numpy as np
import torch

from denno_beta_b200 import cuda as cu

TYPE = {"q4_k": cu.Q4_K, "iq3_xxs": cu.IQ3_XXS, "q6_k": cu.Q6_K, "q8_0": cu.Q8_0, "q5_k": cu.Q5_K}


def _moe(kind, name=None, nt=1, layers=1, gate_up="iq3_xxs", down=None, every=0, e=2048, ff=512, ne=512, k=10, zipf=0.0, **more):
    """A case on MoE layers.  every > 0: each `every`-th layer has Q4_K experts.  zipf: skew of the router's bias."""
    case = dict(kind=kind, nt=nt, layers=layers, gate_up=gate_up, down=down or gate_up, every=every, e=e, ff=ff, ne=ne, k=k, zipf=zipf, **more)
    return dict(case, name=name) if name else case


def _gemv(name=None, ty="q4_k", k=4096, n=4096, count=1, nvec=1, where="dev"):
    case = dict(kind="gemv", ty=ty, k=k, n=n, count=count, nvec=nvec, where=where)
    return dict(case, name=name) if name else case


def listed():
    return [
        # One token, layer by layer with host buffers: an engine whose attention runs elsewhere (the smallest call).
        _moe("block", "token, host buffers", layers=8, where="host"),
        # One token through a resident stack, five layers of IQ3_XXS for each one of Q4_K: single-user decode.
        _moe("stack", "token, stack", layers=12, every=6),
        # Continuous batching at 8 and at 32 sequences, the same mix of layers.
        _moe("block", "batch of 8", nt=8, layers=6, every=6, where="dev"),
        _moe("block", "batch of 32", nt=32, layers=6, every=6, where="dev"),
        # A short prompt on a checkpoint that mixes formats: Q4_K gate and up, Q6_K down.
        _moe("block", "prompt of 77, Q4_K and Q6_K", nt=77, layers=2, gate_up="q4_k", down="q6_k", zipf=1.1, where="dev"),
        # A full prompt chunk under a skewed router, in the two main formats.
        _moe("block", "chunk of 512, Q4_K", nt=512, layers=2, gate_up="q4_k", zipf=1.1, where="dev"),
        _moe("block", "chunk of 512, IQ3_XXS", nt=512, layers=2, zipf=1.1, where="dev"),
        # A long prompt: one layer's 27 chunks of 512 and the ragged last one.
        _moe("prompt", "prompt of 14018", nt=14018, gate_up="q4_k", zipf=1.1, chunk=512),
        # The dense matrices of a quantised model, one token: square projections, and the output head.
        _gemv("gemv 4096 x 4096, Q4_K", count=32),
        _gemv("gemv 65536 x 4096, Q8_0", ty="q8_0", n=65536),
        # The engine routes for itself and hands over the selection (speculative decoding: a few tokens).
        _moe("experts", "4 tokens, selection given", nt=4, layers=4),
        # One token through hyper-connection layers: four residual streams, a gate of rank 320.
        _moe("hyper", "token, hyper-connections", layers=4, hc=4, rank=320),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["block", "block", "block", "block", "stack", "prompt", "gemv", "gemv", "experts", "hyper"])
    if kind == "gemv":
        k = 256 * rng.randint(2, 24)
        n = _log(rng, 300, 65536)
        return _gemv(ty=rng.choice(sorted(TYPE)), k=k, n=n, count=max(1, min(32, (64 << 20) // (k * n))), nvec=rng.choice([1, 1, 1, rng.randint(2, 8)]),
                     where=rng.choice(["dev", "dev", "host"]) if k * n <= 32 << 20 else "dev")
    shape = dict(e=rng.choice([1024, 2048, 2048, 2048]), ff=rng.choice([512, 512, 512, 768]), ne=rng.choice([64, 128, 256, 512, 512]), k=rng.randint(4, 10))
    form = rng.choice([dict(gate_up="iq3_xxs"), dict(gate_up="iq3_xxs"), dict(gate_up="q4_k"), dict(gate_up="q4_k"), dict(gate_up="q4_k", down="q6_k"),
                       dict(gate_up="q8_0"), dict(gate_up="q5_k", down="q6_k")])
    if kind == "stack":
        return _moe("stack", layers=rng.randint(3, 12), every=rng.choice([0, 3, 6]), **shape)
    if kind == "prompt":
        return _moe("prompt", nt=_log(rng, 600, 9000), gate_up=rng.choice(["q4_k", "iq3_xxs"]), zipf=1.1, chunk=512, **shape)
    if kind == "experts":
        return _moe("experts", nt=_log(rng, 1, 12), layers=4, **form, **shape)
    if kind == "hyper":
        return _moe("hyper", nt=_log(rng, 1, 40), layers=2, hc=rng.choice([2, 4]), rank=32 * rng.randint(2, 10), **shape)
    nt = _log(rng, 1, 700)
    return _moe("block", nt=nt, layers=6 if nt < 16 else 2, zipf=1.1 if nt > 64 else 0.0, where=rng.choice(["dev", "dev", "host"]), **form, **shape)


# ---- preparation -------------------------------------------------------------------------------------------------------

_stream = []


def _on_stream():
    """The one stream that all contexts of this process work on, as those of a program around torch would."""
    if not _stream:
        _stream.append(torch.cuda.Stream())
    return _stream[0]


class State:
    """A context with its registered weights, and the buffers of a pass; gives the context's memory back when it goes."""

    def __init__(self, case):
        self.case = case
        self.ctx = cu.CudaCtx(0)
        self.ctx.set_stream(_on_stream().cuda_stream)
        self.layers = range(case.get("layers", 0))

    def __del__(self):
        if getattr(self, "ctx", None) is not None:
            self.ctx.close()


def _layer_types(case, layer):
    if case["every"] and layer % case["every"] == case["every"] - 1:
        return "q4_k", "q4_k"
    return case["gate_up"], case["down"]


def _normal(gen, sigma, *shape):
    return torch.randn(*shape, generator=gen, device="cuda") * sigma


def _host(t):
    return np.ascontiguousarray(t.cpu().numpy())


def _zipf_bias(gen, s, ne):
    """-s * ln(rank + 1) over a random order of the experts."""
    ranks = torch.randperm(ne, generator=gen, device="cuda").float()
    return -s * torch.log(ranks + 1.0)


def _register_layer(ctx, case, gen, layer, seed):
    e, ff, ne = case["e"], case["ff"], case["ne"]
    gate_up, down = (TYPE[t] for t in _layer_types(case, layer))
    for matrix, ty, n_in, n_out, n in ((cu.GATE, gate_up, e, ff, ne), (cu.UP, gate_up, e, ff, ne), (cu.DOWN, down, ff, e, ne),
                                       (cu.SHARED_GATE, gate_up, e, ff, 1), (cu.SHARED_UP, gate_up, e, ff, 1), (cu.SHARED_DOWN, down, ff, e, 1)):
        if not ctx.synth_experts(layer, matrix, ty, n_in, n_out, n, seed):
            raise RuntimeError("synth_experts declined")
    # hyper-connection layers normalise in the mix; every other block has its own RMSNorm
    norm = None if case["kind"] == "hyper" else _host(1.0 + _normal(gen, 0.1, e))
    bias = _host(_zipf_bias(gen, case["zipf"], ne)) if case["zipf"] else None
    ctx.register_router(layer, _host(_normal(gen, 0.02, ne, e)), bias, norm)


def _blocks(gen, ty, count):
    """`count` random blocks of a format: uniform payload, half-precision scales |N(0,1)| * 0.01 (0.02 for IQ3_XXS)."""
    size = cu.TYPE_SIZE[TYPE[ty]]
    b = torch.randint(0, 256, (count, size), dtype=torch.uint8, generator=gen, device="cuda")
    at = {"q4_k": (0, 2), "q5_k": (0, 2), "q6_k": (208,), "q8_0": (0,), "iq3_xxs": (0,)}[ty]
    if ty == "q6_k":
        b[:, 192:208] = ((b[:, 192:208].int() & 63) - 32).to(torch.int8).view(torch.uint8)
    for a in at:
        d = (torch.randn(count, 1, generator=gen, device="cuda").abs() * (0.02 if ty == "iq3_xxs" else 0.01)).half()
        b[:, a:a + 2] = d.view(torch.uint8)
    return b


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    s = State(case)
    if case["kind"] == "gemv":
        _prepare_gemv(s, gen)
    else:
        _prepare_moe(s, gen, seed)
    torch.cuda.synchronize()
    return s


def _prepare_gemv(s, gen):
    case, ctx = s.case, s.ctx
    ty, k, n, count, nvec = case["ty"], case["k"], case["n"], case["count"], case["nvec"]
    s.w = [_blocks(gen, ty, n * k // cu.BLOCK_ELEMS[TYPE[ty]]) for _ in range(count)]
    s.x = _normal(gen, 1.0, count, nvec, k)
    s.out = torch.empty(count, nvec, n, device="cuda")
    if case["where"] == "host":
        for i, w in enumerate(s.w):
            if not ctx.register_matrix(i, TYPE[ty], w.cpu().numpy().reshape(-1), k, n):
                raise RuntimeError("register_matrix declined")
        s.w = None
        s.x, s.out = _host(s.x), np.empty((count, nvec, n), np.float32)


def _prepare_moe(s, gen, seed):
    case, ctx = s.case, s.ctx
    e, ne, k, nt, n = case["e"], case["ne"], case["k"], case["nt"], len(s.layers)
    if not ctx.moe_config(n, e, case["ff"], ne, k):
        raise RuntimeError("moe_config declined")
    for layer in s.layers:
        _register_layer(ctx, case, gen, layer, seed)
    if case["kind"] == "experts":
        s.x = _host(_normal(gen, 1.0, n, nt, e))
        picks = torch.rand(n, nt, ne, generator=gen, device="cuda").topk(k).indices.sort().values
        s.sels = np.ascontiguousarray(picks.cpu().numpy().astype(np.int32))
        w = torch.rand(n, nt, k, generator=gen, device="cuda") + 0.1
        s.wts = _host(w / w.sum(-1, keepdim=True))
    elif case["kind"] == "hyper":
        hc, rank = case["hc"], case["rank"]
        for layer in s.layers:
            ctx.register_hc(layer, hc, rank, _host(1.0 + _normal(gen, 0.1, hc * e)), _host(_normal(gen, (hc * e) ** -0.5, (rank + hc) * hc * e)),
                            _host(_normal(gen, 2.0 * rank ** -0.5, hc * e * rank)))
        s.x = _host(_normal(gen, 1.0, n, nt, hc, e))
    elif case.get("where") == "host":
        s.x = _host(_normal(gen, 1.0, n, nt, e))
        s.out = np.empty((n, nt, e), np.float32)
        s.ptrs = [(cu.host_ptr(s.x[i]), cu.host_ptr(s.out[i])) for i in s.layers]
    else:
        s.x = _normal(gen, 1.0, n, nt, e)
        s.out = torch.empty(n, nt, e, device="cuda")


# ---- a pass ------------------------------------------------------------------------------------------------------------

def _done(ok):
    if ok is None or ok is False:
        raise RuntimeError("the library declined the call")
    return ok


def run(s):
    return RUN[s.case["kind"]](s, s.case, s.ctx)


def _run_gemv(s, case, ctx):
    if case["where"] == "host":
        for i in range(case["count"]):
            for v in range(case["nvec"]):
                _done(ctx.gemv(i, s.x[i, v], s.out[i, v]))
        return s.out
    ty, k, n, nvec = TYPE[case["ty"]], case["k"], case["n"], case["nvec"]
    x, out = s.x.data_ptr(), s.out.data_ptr()
    for i, w in enumerate(s.w):
        _done(ctx.gemv_dev(ty, w.data_ptr(), k, n, x + 4 * i * nvec * k, out + 4 * i * nvec * n, nvec))
    return s.out


def _run_block(s, case, ctx):
    nt = case["nt"]
    if case["where"] == "host":
        for layer in s.layers:
            _done(ctx.moe_block_into(layer, *s.ptrs[layer], nt))
        return s.out
    x, out, step = s.x.data_ptr(), s.out.data_ptr(), 4 * nt * case["e"]
    for layer in s.layers:
        _done(ctx.moe_block_dev(layer, x + layer * step, nt, out + layer * step))
    return s.out


def _run_stack(s, case, ctx):
    nbytes = 4 * case["nt"] * case["e"]
    ctx.dev_copy(s.out.data_ptr(), s.x.data_ptr(), nbytes)  # the token's embedding; the stack works in place
    _done(ctx.moe_stack_dev(s.out.data_ptr(), case["nt"]))
    return s.out[0]


def _run_prompt(s, case, ctx):
    nt, chunk, row = case["nt"], case["chunk"], 4 * case["e"]
    x, out = s.x.data_ptr(), s.out.data_ptr()
    for layer in s.layers:
        for t in range(0, nt, chunk):
            _done(ctx.moe_block_dev(layer, x + t * row, min(chunk, nt - t), out + t * row))
    return s.out


def _run_experts(s, case, ctx):
    return [_done(ctx.moe_experts(layer, s.x[layer], s.sels[layer], s.wts[layer])) for layer in s.layers]


def _run_hyper(s, case, ctx):
    return [_done(ctx.hc_moe_block(layer, s.x[layer])) for layer in s.layers]


RUN = {"gemv": _run_gemv, "block": _run_block, "stack": _run_stack, "prompt": _run_prompt, "experts": _run_experts, "hyper": _run_hyper}


# ---- what a pass needs, and how exact it is ------------------------------------------------------------------------------

def _active(case, nt):
    """Distinct experts that nt tokens select: a sample of the router's scores (variance e * 0.02^2) plus the skewed bias."""
    ne, k = case["ne"], case["k"]
    rng = np.random.RandomState(1)
    if case["kind"] == "experts":
        score = rng.rand(nt, ne)
    else:
        score = rng.randn(nt, ne) * 0.02 * math.sqrt(case["e"]) - case["zipf"] * np.log(1.0 + np.arange(ne))
    return len(np.unique(np.argpartition(-score, k - 1, axis=1)[:, :k]))


def work(case):
    if case["kind"] == "gemv":
        k, n, count, nvec = case["k"], case["n"], case["count"], case["nvec"]
        return {"bytes": count * (n * cu.row_bytes(TYPE[case["ty"]], k) + 4 * nvec * (k + n)), "flops": 2 * count * nvec * k * n}
    e, ff, ne, k, nt = (case[x] for x in ("e", "ff", "ne", "k", "nt"))
    routed = case["kind"] != "experts"
    # a chunk's weights are read once each; activations once in and once out
    sizes = [nt] if case["kind"] != "prompt" else [min(case["chunk"], nt - t) for t in range(0, nt, case["chunk"])]
    found = {size: _active(case, size) for size in set(sizes)}
    active = sum(found[size] + 1 for size in sizes)
    nbytes = flops = 0
    for layer in range(case["layers"]):
        gate_up, down = (TYPE[t] for t in _layer_types(case, layer))
        nbytes += active * (2 * ff * cu.row_bytes(gate_up, e) + e * cu.row_bytes(down, ff)) + 8 * nt * e + len(sizes) * 4 * ne * e * routed
        flops += 6 * nt * (k + 1) * e * ff + 2 * nt * ne * e * routed
        if case["kind"] == "hyper":
            hc, rank = case["hc"], case["rank"]
            nbytes += 4 * hc * e * (2 * rank + hc) + 8 * nt * (hc - 1) * e
            flops += 2 * nt * hc * e * (2 * rank + hc)
    return {"bytes": nbytes, "flops": flops}


def tolerance(case):
    if case["kind"] == "gemv":
        return {"rel": 1e-5, "max": 1e-4}  # one sum of k products in 32 bits
    types = {t for layer in range(case["layers"]) for t in _layer_types(case, layer)}
    if case["kind"] in ("block", "prompt", "hyper") and case["nt"] >= 16 and types <= {"q4_k", "iq3_xxs"}:
        # tensor-core chunks: 16 significant bits per operand (two bf16 parts), 32-bit sums, two GEMMs in a row
        return {"rel": 2e-4, "max": 4e-3}
    # 32-bit operands and sums; a stack carries one layer's rounding through the next ones' normalisation
    return {"rel": 1e-4 if case["kind"] == "stack" else 2e-5, "max": 1e-3}
