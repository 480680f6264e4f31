"""What is timed when this package's speed is looked at: the calls that a program built on it makes, with their inputs.

A case is a dict of plain values. `kind` says which call it is:

  token     chat at batch 1: one token in, the next token's logits out (`PSSAModel.forward_inference`)
  prompt    one prompt read behind a cached prefix: the prefix's carry in, the last token's logits and the new carry out
  batch     the next turns of several conversations, of different lengths, in one call: host ids in, host logits out
            (`prefill_batch`)
  stream    tokens for every lane with ids and logits in device memory (`prefill_batch_dev`): one token per lane is a step
            of a decode loop, many are the prefill of a batch
  sample    one step of scored sampling in the fp32 mode, where tokens have to be the CPU model's (`decode_step_sampled`)
  score     next-token losses of a text under a frozen model (`PSSAModel.score`)
  scan      the recurrence operator alone, device arrays (`scan_states_dev`)
  read      the top-8 memory read alone, device arrays (`memory_read_topk_dev`)
  seam      one block through the host-array operators that stand in for the reference's device seam: projections, SSM,
            memory stage and MLP, each call with numpy arrays in and out

Three model sizes: `small` and `base` are the repository's one-block and twelve-block configurations, `mid` lies between
them with widths that are no tile's multiple and a bank that is not full. Every stream has read `PREFIX` tokens before the
call that is timed: the carry of a fresh stream is all zeros, which no call but a stream's first one meets, and with random
weights the features of the first tokens can nearly cancel, so that their values are mostly rounding.
"""
import math

import numpy as np
import torch

import pssa_b200
from pssa_b200 import _native as N
from pssa_b200 import model as M

RANK = 16  # of the adapter
SIZES = {
    "small": dict(depth=1, vocab=8192, d=192, s=64, k=64, cap=512, count=512),
    "mid": dict(depth=4, vocab=5003, d=384, s=32, k=64, cap=256, count=200),
    "base": dict(depth=12, vocab=16384, d=768, s=64, k=64, cap=512, count=512),
}
TAU = 0.1
PREFIX = 256
MODEL_KINDS = ("token", "prompt", "batch", "stream", "sample", "score")


def listed():
    return [
        # chat at batch 1 on the smallest model: a step is launches and host work
        dict(name="token_small", kind="token", size="small", fp32=False),
        # a prompt for it, in the mode that reproduces the CPU model's tokens
        dict(name="prompt_small_fp32", kind="prompt", size="small", length=512, fp32=True),
        # chat at batch 1 on the large model
        dict(name="token_base", kind="token", size="base", fp32=False),
        # a long document at batch 1
        dict(name="prompt_long", kind="prompt", size="base", length=8192, fp32=False),
        # a server's admission step: a handful of turns, no two of one length
        dict(name="prompts_ragged", kind="batch", size="base", lanes=7, shortest=33, longest=1501, fp32=False),
        # many streams decoding together
        dict(name="decode_256", kind="stream", size="base", lanes=256, length=1, fp32=False),
        # throughput prefill
        dict(name="prefill_32x2048", kind="stream", size="base", lanes=32, length=2048, fp32=False),
        # scored sampling that reproduces the CPU model's tokens
        dict(name="sample_fp32", kind="sample", size="base", streams=16),
        # perplexity of a text
        dict(name="score_2048", kind="score", size="base", length=2048, fp32=False),
        # the recurrence alone on one long sequence of the large model's states
        dict(name="scan_long", kind="scan", lanes=1, length=8191, stride=49152, carry=True),
        # the memory read alone at its own configuration
        dict(name="read_top8", kind="read", rows=262144, dk=128, dv=128, cap=512, count=512),
        # one block for a host program that calls the operators one by one
        dict(name="seam_block", kind="seam", size="small", length=128),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("token", "prompt", "prompt", "batch", "batch", "stream", "stream", "stream", "sample", "score", "scan", "read", "seam"))
    size = rng.choice(("small", "mid", "base"))
    if kind == "token":
        return dict(kind=kind, size=size, fp32=rng.random() < 0.25)
    if kind == "prompt":
        fp32 = rng.random() < 0.25
        return dict(kind=kind, size=size, length=_log(rng, 2, 512 if fp32 else 16384), fp32=fp32)
    if kind == "batch":
        fp32 = rng.random() < 0.25
        longest = _log(rng, 16, 300 if fp32 else 2048)
        return dict(kind=kind, size=size, lanes=_log(rng, 2, 4 if fp32 else 24), shortest=_log(rng, 1, longest), longest=longest, fp32=fp32)
    if kind == "stream":
        if rng.random() < 0.5:
            return dict(kind=kind, size=size, lanes=_log(rng, 2, 512), length=1, fp32=False)
        lanes = _log(rng, 2, 64)
        return dict(kind=kind, size=size, lanes=lanes, length=_log(rng, 16, 65536 // lanes), fp32=False)
    if kind == "sample":
        return dict(kind=kind, size=size, streams=_log(rng, 1, 64))
    if kind == "score":
        return dict(kind=kind, size=size, length=_log(rng, 16, 8192), fp32=False)
    if kind == "scan":
        lanes, stride = _log(rng, 1, 64), _log(rng, 64, 49152)
        return dict(kind=kind, lanes=lanes, length=_log(rng, 16, max(17, min(65536, (1 << 29) // (lanes * stride)))), stride=stride, carry=rng.random() < 0.5)
    if kind == "read":
        cap = rng.choice((128, 256, 512))
        return dict(kind=kind, rows=_log(rng, 1, 262144), dk=rng.choice((64, 128)), dv=rng.choice((64, 128, 192, 768)), cap=cap,
                    count=rng.randint(96, cap))
    return dict(kind="seam", size=rng.choice(("small", "mid")), length=_log(rng, 1, 512))


# ---- inputs

def _normal(gen, scale, *shape):
    return (torch.randn(*shape, device="cuda", generator=gen) * scale).contiguous()


def _uniform(gen, lo, hi, *shape):
    return torch.rand(*shape, device="cuda", generator=gen) * (hi - lo) + lo


def _ball(gen, rows, width):
    """Points of the unit ball with norms below 0.9."""
    x = torch.randn(rows, width, device="cuda", generator=gen)
    return (x / x.norm(dim=1, keepdim=True) * _uniform(gen, 0.0, 0.9, rows, 1)).contiguous()


def _host(x):
    return x.contiguous().cpu().numpy()


def _ids(gen, vocab, n):
    return torch.randint(1, vocab, (n,), device="cuda", generator=gen)


def _block_weights(gen, z):
    d, s, k = z["d"], z["s"], z["k"]
    shapes = {M.W_DELTA: (d, d), M.W_B: (s, d), M.W_C: (s, d), M.W_QX: (k, d), M.W_QH: (k, d), M.W_GATE: (d, d), M.W_PROJ: (d, d),
              M.MLP_W1: (2 * d, d), M.MLP_W2: (d, 2 * d), M.AD_DOWN: (RANK, d), M.AD_UP: (d, RANK), M.AD_CONS: (d, RANK)}
    w = {tid: _normal(gen, 0.02, *shape) for tid, shape in shapes.items()}
    decay = _uniform(gen, 0.9, 0.999, d * s)
    w[M.A_MAT] = torch.log(torch.expm1(-torch.log(decay)))  # exp(-softplus(A)) = decay
    return w


def _bank(gen, z):
    keys = _ball(gen, z["cap"], z["k"])
    return keys, (keys.double() ** 2).sum(1).float(), _normal(gen, 1.0, z["cap"], z["d"])


def _model(gen, z, streams, fp32):
    gpu = pssa_b200.B200Dispatch(0, torch.cuda.current_stream())
    m = pssa_b200.PSSAModel(gpu, z["depth"], z["vocab"], z["d"], z["s"], z["k"], z["cap"], tau_mem=TAU, streams=streams,
                            precision=N.PRECISION_FP32_EXACT if fp32 else N.PRECISION_BF16)
    for tid in (M.EMBED, M.UNEMBED):
        m.set_tensor(-1, tid, _host(_normal(gen, 0.02, z["vocab"], z["d"])))
    for layer in range(z["depth"]):
        for tid, w in _block_weights(gen, z).items():
            m.set_tensor(layer, tid, _host(w))
        keys, norm_sq, values = _bank(gen, z)
        m.set_bank(layer, _host(keys), _host(norm_sq), _host(values), z["count"])
    return m


def _lengths(case):
    """Prompt lengths of a batch: the shortest and the longest, and others between them."""
    rng = np.random.default_rng(case["lanes"] * 100003 + case["longest"])
    mid = rng.integers(case["shortest"], case["longest"] + 1, case["lanes"] - 2)
    return [case["longest"], case["shortest"]] + [int(x) for x in mid]


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    kind = case["kind"]
    if kind in MODEL_KINDS:
        return _prepare_model(case, gen)
    if kind == "scan":
        lanes, length, stride = case["lanes"], case["length"], case["stride"]
        a = _uniform(gen, 0.9, 0.999, lanes, length, stride)
        b = _normal(gen, 1.0, lanes, length, stride)
        h0 = _normal(gen, 1.0, lanes, stride) if case["carry"] else None
        return dict(case=case, gpu=pssa_b200.B200Dispatch(0, torch.cuda.current_stream()), a=a, b=b, h0=h0, h=torch.empty_like(a),
                    last=torch.empty(lanes, stride, device="cuda"))
    if kind == "read":
        rows, dk, dv, cap = case["rows"], case["dk"], case["dv"], case["cap"]
        keys = _ball(gen, cap, dk)
        return dict(case=case, gpu=pssa_b200.B200Dispatch(0, torch.cuda.current_stream()), q=_ball(gen, rows, dk), keys=keys,
                    norm_sq=(keys.double() ** 2).sum(1).float(), values=_normal(gen, 1.0, cap, dv),
                    m=torch.empty(rows, dv, device="cuda"), slots=torch.empty(rows, 8, dtype=torch.int32, device="cuda"),
                    weights=torch.empty(rows, 8, device="cuda"))
    z, t = SIZES[case["size"]], case["length"]
    w = {tid: _host(x) for tid, x in _block_weights(gen, z).items()}
    w[M.A_MAT] = (-np.log1p(np.exp(w[M.A_MAT].astype(np.float64)))).astype(np.float32)  # the rates the operator takes
    keys, norm_sq, values = (_host(x) for x in _bank(gen, z))
    x = torch.randn(t, z["d"], device="cuda", generator=gen)
    x = x / x.square().mean(1, keepdim=True).sqrt()
    carry = _host(_normal(gen, 0.1, z["d"] * z["s"]))
    return dict(case=case, gpu=pssa_b200.B200Dispatch(0), w=w, keys=keys, norm_sq=norm_sq, values=values, x=_host(x), carry=carry)


def _prepare_model(case, gen):
    z, kind = SIZES[case["size"]], case["kind"]
    lanes = case.get("lanes") or case.get("streams") or 1
    m = _model(gen, z, lanes, case.get("fp32", kind == "sample"))
    st = dict(case=case, model=m)
    if kind != "score":
        prefix = _host(_ids(gen, z["vocab"], lanes * PREFIX)).astype(np.uint64).reshape(lanes, PREFIX)
        m.prefill_batch(list(prefix), want_logits=False)
    if kind == "token":
        st["ids"] = [int(i) for i in _ids(gen, z["vocab"], 1)]
    elif kind in ("prompt", "score"):
        st["prefix"] = m.copy_recurrent_state_to(0) if kind == "prompt" else None
        ids = _host(_ids(gen, z["vocab"], case["length"] + 1)).astype(np.uint64)
        st["ids"], st["targets"] = ids[:-1].copy(), ids[1:].copy()
    elif kind == "batch":
        st["ids"] = [_host(_ids(gen, z["vocab"], n)).astype(np.uint64) for n in _lengths(case)]
    elif kind == "sample":
        st["ids"] = _host(_ids(gen, z["vocab"], lanes)).astype(np.uint64)
        for i in range(lanes):
            m.sampler_seed(i, 1337 + i)
            m.sampler_push(_host(_ids(gen, z["vocab"], 24)).astype(np.uint64), i)
    else:
        rows = lanes * case["length"]
        st["ids"] = _ids(gen, z["vocab"], rows).to(torch.int32)
        st["offsets"] = np.arange(lanes, dtype=np.uint32) * case["length"]
        st["lengths"] = np.full(lanes, case["length"], np.uint32)
        st["logits"] = torch.empty(lanes, z["vocab"], device="cuda")
    return st


# ---- one pass

def run(st):
    kind = st["case"]["kind"]
    if kind == "token":
        return st["model"].forward_inference(st["ids"][0])
    if kind == "prompt":
        m = st["model"]
        m.copy_recurrent_state_from(st["prefix"], 0)
        _, logits = m.prefill_inference(st["ids"])
        return logits, m.copy_recurrent_state_to(0)
    if kind == "batch":  # the carries run on: a call continues the call before it
        return st["model"].prefill_batch(st["ids"])[0]
    if kind == "stream":  # and here
        st["model"].prefill_batch_dev(st["ids"], st["offsets"], st["lengths"], None, st["logits"])
        return st["logits"]
    if kind == "sample":
        st["ids"], confidence = st["model"].decode_step_sampled(st["ids"], want_confidence=True)
        return st["ids"], confidence
    if kind == "score":
        m = st["model"]
        m.reset_recurrent_state(0)
        return m.score(st["ids"], st["targets"])
    c, gpu = st["case"], st["gpu"]
    if kind == "scan":
        gpu.scan_states_dev(st["a"], st["b"], st["h0"], st["h"], st["last"], c["lanes"], c["length"], c["stride"])
        return st["h"], st["last"]
    if kind == "read":
        gpu.memory_read_topk_dev(st["q"], st["keys"], st["norm_sq"], st["values"], c["rows"], c["dk"], c["dv"], c["cap"], c["count"], TAU, 8,
                                 st["m"], st["slots"], st["weights"], q_is_euclidean=False)
        return st["m"], st["slots"], st["weights"]
    return _run_seam(st)


def _run_seam(st):
    z, t, gpu, w, x = SIZES[st["case"]["size"]], st["case"]["length"], st["gpu"], st["w"], st["x"]
    d, s, k = z["d"], z["s"], z["k"]
    delta = gpu.dispatch_gemm(x, w[M.W_DELTA], t, d, d, 1, epilogue=N.EPI_SOFTPLUS)
    b = gpu.dispatch_gemm(x, w[M.W_B], t, s, d, 1)
    c = gpu.dispatch_gemm(x, w[M.W_C], t, s, d, 1)
    y, states = np.empty(t * d, np.float32), np.empty((t + 1) * d * s, np.float32)
    gpu.ssm_forward(delta, b, x, w[M.A_MAT], c, st["carry"], t, d, s, states=states, y_ssm=y)
    mem = gpu.memory_forward(x, y, w[M.W_QX], w[M.W_QH], w[M.W_GATE], w[M.W_PROJ], st["keys"], st["norm_sq"], st["values"], t, d, k, d,
                             z["cap"], z["count"], TAU)
    zr = mem["m_inj"].reshape(t, d) + y.reshape(t, d) / np.float32(math.sqrt(s))
    h = gpu.dispatch_gemm(zr, w[M.MLP_W1], t, 2 * d, d, 1, epilogue=N.EPI_SILU)
    out = gpu.dispatch_gemm(h, w[M.MLP_W2], t, d, 2 * d, 1)
    return out, y, states, mem


# ---- what a pass cannot do without

def _block_params(z):
    d, s, k = z["d"], z["s"], z["k"]
    return 2 * d * d + 2 * s * d + k * d + RANK * d + k * d + d * d + 4 * d * d + RANK * d


def _model_work(case):
    """Weights, rates and banks once at the mode's width, the carries in and out, ids in, results out; two operations per weight and row,
    the memory read's two contractions and the recurrence."""
    z, kind = SIZES[case["size"]], case["kind"]
    fp32 = case.get("fp32", kind == "sample")
    d, s, v = z["d"], z["s"], z["vocab"]
    lanes = case.get("lanes") or case.get("streams") or 1
    rows = sum(_lengths(case)) if kind == "batch" else lanes * case.get("length", 1)
    heads = rows if kind == "score" else lanes
    width = 4 if fp32 else 2
    weights = (z["depth"] * (_block_params(z) + z["count"] * (z["k"] + d)) + v * d) * width + z["depth"] * d * s * 4 + min(rows, v) * d * 4
    carries = lanes * z["depth"] * d * s * 4 * (1 if kind == "score" else 2)
    results = {"score": 4 * rows, "sample": 12 * lanes}.get(kind, 4 * v * heads)
    per_row = 2 * _block_params(z) + 2 * z["count"] * (z["k"] + d) + 6 * d * s
    return {"bytes": weights + carries + results + 4 * rows, "flops": rows * z["depth"] * per_row + heads * 2 * v * d}


def work(case):
    kind = case["kind"]
    if kind in MODEL_KINDS:
        return _model_work(case)
    if kind == "scan":
        n, row = case["lanes"] * case["length"] * case["stride"], case["lanes"] * case["stride"]
        return {"bytes": 12 * n + 4 * row * (2 if case["carry"] else 1), "flops": 2 * n}
    if kind == "read":
        rows, dk, dv, cap = case["rows"], case["dk"], case["dv"], case["cap"]
        return {"bytes": 4 * (rows * (dk + dv + 16) + cap * (dk + dv + 1)), "flops": rows * (3 * dk * case["count"] + 16 * dv)}
    z, t = SIZES[case["size"]], case["length"]
    d, s, k, cap = z["d"], z["s"], z["k"], z["cap"]
    ins = 7 * d * d + 2 * s * d + 2 * k * d + 2 * d * s + cap * (k + 1 + d) + t * d
    outs = t * (d + d + d * s) + d * s + t * (2 * k + 1 + cap + 4 * d)
    return {"bytes": 4 * (ins + outs), "flops": t * (2 * (7 * d * d + 2 * s * d + 2 * k * d) + 6 * d * s + 2 * z["count"] * (k + d))}


def tolerance(case):
    kind = case["kind"]
    if kind in MODEL_KINDS and not case.get("fp32", kind == "sample"):
        # bf16 operands: a rounding of 2^-9 in the inputs of every product. Against the fp32 mode that is 5e-3 of the logits after
        # one block, 8e-3 after four and 1.5e-2 after twelve; a loss is near log(vocab) and moves by its few logits' error.
        return {"rel": 3e-4} if kind == "score" else {"rel": 2e-2 if case["size"] == "base" else 1e-2}
    return {"rel": 1e-5}
