"""The work a user of this framework has it do, as cases that can be timed and compared.

Five kinds, each through the call a program makes:

  linear    one ``ADEKernelLinear.forward``: the factored path up to 128 token rows, the reconstructed path above;
  decode    eight steps of token-by-token decoding of a LLaMA-architecture model whose linear modules all carry a
            delta: static KV cache, the step captured once in a CUDA graph (as ``GreedyGraphDecoder`` does) and replayed;
  prefill   one forward of such a model over a prompt, as transformers runs it;
  merge     ``recon_int4``: a module's delta folded into its base weight, once;
  compress  ``compress_module`` on the GPU and ``pack_int4`` of the result: from a truncated SVD to what the kernels read.

Sizes are those of the 7B and 13B LLaMA architectures in ``ade_b200.synth`` (hidden 4096 / 5120, MLP 11008 / 13824),
of the small ragged modules in the tests, and random ones between them.  Models have eight of their architecture's
layers: every layer is the same work, and the logits of two correct implementations still agree (in a deep stack of random
weights a rounding difference of the residual stream grows from layer to layer).
"""
from __future__ import annotations

import math

import torch

from ade_b200 import kernels, quantization, synth
from ade_b200.serving import ADEKernelLinear

DEVICE = "cuda"
STEPS = 8                       # decode steps of one pass
VOCAB = 32000


def listed():
    return [
        # the smallest call: a narrow, ragged projection on three token rows (speculative drafts, small models)
        {"name": "linear_1000x2048_r384_t3", "kind": "linear", "M": 1000, "N": 2048, "r": 384, "T": 3},
        # an attention projection with the 16 rows of a small batch: the framework's single-module configuration
        {"name": "linear_4096x4096_r256_t16", "kind": "linear", "M": 4096, "N": 4096, "r": 256, "T": 16},
        # a ragged module and row count in the middle of the factored range, at a high rank
        {"name": "linear_5000x5120_r896_t40", "kind": "linear", "M": 5000, "N": 5120, "r": 896, "T": 40},
        # a short prompt (100 tokens) through an MLP down projection: the upper end of the factored range
        {"name": "linear_4096x11008_r512_t100", "kind": "linear", "M": 4096, "N": 11008, "r": 512, "T": 100},
        # a long prompt through an MLP gate projection: the reconstructed path
        {"name": "linear_11008x4096_r512_t2048", "kind": "linear", "M": 11008, "N": 4096, "r": 512, "T": 2048},
        # one user's generation: latency per token
        {"name": "decode_7b_b1", "kind": "decode", "arch": "7b", "layers": 8, "batch": 1, "ctx": 64},
        # eight users behind 512-token prompts
        {"name": "decode_13b_b8", "kind": "decode", "arch": "13b", "layers": 8, "batch": 8, "ctx": 512},
        # a serving batch of 32, above the range in which the base GEMM is part of the factored launch
        {"name": "decode_7b_b32", "kind": "decode", "arch": "7b", "layers": 8, "batch": 32, "ctx": 260},
        # a short prompt: time to the first token
        {"name": "prefill_7b_1x64", "kind": "prefill", "arch": "7b", "layers": 8, "batch": 1, "prompt": 64},
        # four 500-token prompts: the reconstructed path in every module
        {"name": "prefill_7b_4x500", "kind": "prefill", "arch": "7b", "layers": 8, "batch": 4, "prompt": 500},
        # merging a delta into its base model, the largest module at the highest usual rank
        {"name": "merge_13824x5120_r1024", "kind": "merge", "M": 13824, "N": 5120, "r": 1024},
        # producing a delta: quantising the two factors of an MLP module and packing them for the kernels
        {"name": "compress_11008x4096_r512", "kind": "compress", "M": 11008, "N": 4096, "r": 512},
    ]


def _log(rng, lo, hi):
    """A whole number in [lo, hi], spread evenly over its logarithm."""
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["linear", "linear", "linear", "linear", "decode", "decode", "prefill", "merge", "merge", "compress"])
    if kind == "linear":
        return {"kind": kind, "M": _log(rng, 500, 13824), "N": 128 * _log(rng, 8, 108), "r": 128 * rng.randint(1, 8), "T": _log(rng, 1, 2500)}
    if kind == "decode":
        return {"kind": kind, "arch": rng.choice(["7b", "13b"]), "layers": rng.randint(2, 8), "batch": _log(rng, 1, 48), "ctx": _log(rng, 20, 600)}
    if kind == "prefill":
        return {"kind": kind, "arch": rng.choice(["7b", "13b"]), "layers": rng.randint(2, 8), "batch": rng.randint(1, 3), "prompt": _log(rng, 20, 700)}
    M, N, r = _log(rng, 500, 13824), 128 * _log(rng, 8, 108), 128 * rng.randint(1, 8)
    return {"kind": kind, "M": M, "N": N, "r": r}


# ------------------------------------------------------------------------------------ state
def _gen(seed):
    return torch.Generator(device=DEVICE).manual_seed(seed)


def _module(M, N, r, seed):
    """Base weight ~ N(0, 0.02^2) and packed delta whose entries are about a tenth of it."""
    g = _gen(seed)
    W = (torch.randn(M, N, generator=g, device=DEVICE) * 0.02).to(torch.bfloat16)
    packed = synth.random_packed(M, N, r, seed + 1, DEVICE, on_device=True)
    for k in ("U_scale", "Vt_scale"):
        packed[k] = packed[k] * 3.0
    return W, packed


def _model(case, seed):
    """The architecture with random weights and a delta on every linear module.  Embeddings are scaled up so that a layer
    adds a small part to the residual stream, as in a trained model."""
    model, _, _ = synth.synthetic_llama(case["arch"], layers=case["layers"], seed=seed, device=DEVICE, vocab=VOCAB)
    with torch.no_grad():
        model.model.embed_tokens.weight.mul_(800.0)
    return model


def _decode_state(case, seed):
    from transformers import StaticCache

    batch, ctx = case["batch"], case["ctx"]
    model = _model(case, seed)
    g = _gen(seed + 1)
    prompt = torch.randint(0, VOCAB, (batch, ctx), generator=g, device=DEVICE)
    fed = torch.randint(0, VOCAB, (STEPS, batch, 1), generator=g, device=DEVICE)
    cache = StaticCache(config=model.config, max_cache_len=ctx + STEPS + 1)
    tok = torch.zeros(batch, 1, dtype=torch.long, device=DEVICE)
    pos = torch.zeros(1, dtype=torch.long, device=DEVICE)

    def step():
        return model(input_ids=tok, past_key_values=cache, cache_position=pos, use_cache=True).logits

    def rewind():
        pos.fill_(ctx)
        for layer in cache.layers:
            layer.cumulative_length.fill_(ctx)

    with torch.no_grad():
        model(input_ids=prompt, past_key_values=cache, cache_position=torch.arange(ctx, device=DEVICE), use_cache=True, logits_to_keep=1)
        rewind()
        side = torch.cuda.Stream()
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(side):
            for _ in range(2):
                step()
        torch.cuda.current_stream().wait_stream(side)
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            logits = step()
    out = torch.empty(STEPS, batch, VOCAB, dtype=logits.dtype, device=DEVICE)
    return {"model": model, "cache": cache, "graph": graph, "tok": tok, "pos": pos, "fed": fed, "logits": logits, "rewind": rewind, "out": out}


def prepare(case, seed):
    kind = case["kind"]
    if kind == "linear":
        W, packed = _module(case["M"], case["N"], case["r"], seed)
        x = torch.randn(case["T"], case["N"], generator=_gen(seed + 2), device=DEVICE).to(torch.bfloat16)
        return {"kind": kind, "lin": ADEKernelLinear(W, packed), "x": x}
    if kind == "decode":
        return dict(_decode_state(case, seed), kind=kind)
    if kind == "prefill":
        model = _model(case, seed)
        ids = torch.randint(0, VOCAB, (case["batch"], case["prompt"]), generator=_gen(seed + 1), device=DEVICE)
        return {"kind": kind, "model": model, "ids": ids}
    if kind == "merge":
        W, packed = _module(case["M"], case["N"], case["r"], seed)
        return {"kind": kind, "W": W, "p4": kernels.pack_int4(packed)}
    # factors as a truncated SVD has them: columns of about unit length, singular values that fall off
    M, N, r = case["M"], case["N"], case["r"]
    g = _gen(seed)
    U = torch.randn(M, r, generator=g, device=DEVICE) / math.sqrt(M)
    V = torch.randn(N, r, generator=g, device=DEVICE) / math.sqrt(N)
    S = 1.5 * torch.exp(-3.0 * torch.arange(r, device=DEVICE) / r) + 0.1 * torch.rand(r, generator=g, device=DEVICE)
    return {"kind": kind, "U": U, "S": S, "V": V, "seed": seed}


# ------------------------------------------------------------------------------------ one pass
def run(state):
    kind = state["kind"]
    if kind == "linear":
        return state["lin"](state["x"])
    if kind == "decode":
        state["rewind"]()
        for i in range(STEPS):
            state["tok"].copy_(state["fed"][i])
            state["graph"].replay()
            state["out"][i].copy_(state["logits"][:, -1])
            state["pos"].add_(1)
        return state["out"]
    if kind == "prefill":
        with torch.no_grad():
            out = state["model"](input_ids=state["ids"], use_cache=True)
        last = out.past_key_values.layers[-1]
        return {"logits": out.logits, "keys": last.keys, "values": last.values}
    if kind == "merge":
        return kernels.recon_int4(state["p4"], state["W"])
    # the rotation of a rank that is no power of two is drawn from a seeded generator, the same for both factors
    packed = quantization.compress_module(state["U"], state["S"], state["V"], generator=torch.Generator().manual_seed(state["seed"]),
                                          keep_device=True)
    stored = kernels.pack_int4(packed)
    return {"packed": packed, "stored": {k: stored[k] for k in kernels.STORED_KEYS}}


# ------------------------------------------------------------------------------------ what a pass cannot do without
def _linear_work(M, N, r, T):
    """(bytes of weights and delta, flops) of one module on T token rows: the cheaper of the two orders of the product."""
    ng = r // 128
    stream = 2.0 * M * N + (M + N) * r / 2.0 + 2.5 * (M + N) * ng
    return stream, 2.0 * M * N * T + min(2.0 * (M + N) * r * T, 2.0 * M * N * r)


def _model_work(case, rows, steps, positions):
    """(bytes, flops) of `steps` forwards over `rows` token rows each; `positions`: cached positions read per row and step."""
    kw = synth.LLAMA_ARCH[case["arch"]]
    h, inter, layers = kw["hidden_size"], kw["intermediate_size"], case["layers"]
    shapes = [(h, h)] * 4 + [(inter, h)] * 2 + [(h, inter)]
    mean_rank = 512              # what the 1/16 bit budget leaves on average
    stream = flops = 0.0
    for M, N in shapes:
        b, f = _linear_work(M, N, mean_rank, rows)
        stream, flops = stream + b, flops + f
    stream, flops = stream * layers, flops * layers
    stream += 2.0 * VOCAB * h + 2.0 * 2.0 * rows * positions * h * layers + 2.0 * rows * VOCAB
    flops += 2.0 * VOCAB * h * rows + 4.0 * rows * positions * h * layers
    return {"bytes": steps * stream, "flops": steps * flops}


def work(case):
    kind = case["kind"]
    if kind == "decode":
        return _model_work(case, case["batch"], STEPS, case["ctx"] + STEPS / 2)
    if kind == "prefill":
        w = _model_work(case, case["batch"] * case["prompt"], 1, 0)
        kw = synth.LLAMA_ARCH[case["arch"]]
        attention = 2.0 * case["batch"] * case["prompt"] ** 2 * kw["hidden_size"] * case["layers"]        # causal half of q K^T and P V
        return {"bytes": w["bytes"], "flops": w["flops"] + attention}
    M, N, r = case["M"], case["N"], case["r"]
    ng = r // 128
    if kind == "linear":
        stream, flops = _linear_work(M, N, r, case["T"])
        return {"bytes": stream + 2.0 * case["T"] * (M + N), "flops": flops}
    if kind == "merge":
        return {"bytes": 4.0 * M * N + (M + N) * r / 2.0 + 2.5 * (M + N) * ng, "flops": 2.0 * M * N * r}
    # float32 factors in; codes, scales and zero-points out, and the stored form (codes of V in two orders)
    rotate = math.log2(r) if r & (r - 1) == 0 else 2.0 * r
    return {"bytes": (M + N) * r * (4.0 + 1.0 + 0.5) + N * r * 0.5 + (M + N) * ng * 7.0, "flops": (M + N) * r * (rotate + 6.0)}


def tolerance(case):
    kind = case["kind"]
    if kind == "merge":
        return {"rel": 5e-3}
    if kind == "linear":
        return {"rel": 1e-2}
    if kind == "compress":
        # a code or zero-point whose value lies on a rounding boundary may fall to either side when the rotation sums in
        # another order; a packed byte holds two codes
        return {"rel": 1e-3, "max": 0.5, "differ": 2e-3}
    # bfloat16 residual streams of eight layers: two correct implementations differ by about 0.8 % in the logits
    return {"rel": 3e-2}
