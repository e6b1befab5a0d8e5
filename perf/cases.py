"""Workloads of this library as a user's program meets them, in one place: what is timed, what a pass returns and how
far two correct implementations may differ.

Five kinds of work, all through the public entry points:

* ``decode``: one token for every sequence (``RWKV7ForCausalLM.rwkv7_forward_token``), the inner loop of generation;
* ``serve``: the same step with the states in a slot pool (``RWKV7StatePool.decode``), what a server calls;
* ``prefill``: a prompt (``forward``, or ``rwkv7_prefill_chunks`` with the tensor-core scan for long batched prompts);
* ``scan``: the WKV-7 recurrence over a sequence on its own (``self_chunk_rwkv7``), what a host that keeps its own
  layers calls;
* ``a8w8``: one int8 x int8 projection over the rows of a prompt chunk (``A8W8Linear``).

Model shapes are the three of the benchmark (random weights of those sizes).
"""
import math

import torch

import hf_adapter_b200 as hb

DEV = "cuda"
VOCAB = 65536
# name: layers, width, heads, FFN width
SHAPES = {"0.1B": (12, 768, 12, 3072), "2.9B": (32, 2560, 40, 10240), "7.2B": (32, 4096, 64, 16384)}
RANKS = dict(decay_low_rank_dim=64, a_low_rank_dim=64, v_low_rank_dim=32, gate_low_rank_dim=128)
DTYPES = {"fp32": torch.float32, "fp16": torch.float16, "bf16": torch.bfloat16}
# weight formats each shape is run with: (weights, activation type)
FORMATS = {"0.1B": (("dense", "bf16"), ("dense", "fp16"), ("dense", "fp32")),
           "2.9B": (("w8", "fp16"), ("dense", "fp16")),
           "7.2B": (("mm4", "fp16"),)}
PROMPT = 16  # tokens each sequence has seen before a decode step
MAX_PREFILL = 64 * 512  # tokens of the largest prefill pass


def _model_case(kind, shape, weights, dtype, **more):
    return dict(kind=kind, shape=shape, weights=weights, dtype=dtype, **more)


def listed():
    return [
        # the smallest call: one user, the small model in the bf16 of its checkpoint; launches and latency are all there is
        dict(_model_case("decode", "0.1B", "dense", "bf16", state="fp32", batch=1), name="decode-0.1B-bf16-b1"),
        # interactive chat: one user on the large int4 model
        dict(_model_case("decode", "7.2B", "mm4", "fp16", state="fp32", batch=1), name="decode-7.2B-mm4-b1"),
        # the headline configuration: 64 concurrent sequences
        dict(_model_case("decode", "7.2B", "mm4", "fp16", state="fp32", batch=64), name="decode-7.2B-mm4-b64"),
        # bulk generation: 256 concurrent sequences
        dict(_model_case("decode", "7.2B", "mm4", "fp16", state="fp32", batch=256), name="decode-7.2B-mm4-b256"),
        # an unquantised model, a handful of users
        dict(_model_case("decode", "2.9B", "dense", "fp16", state="fp32", batch=8), name="decode-2.9B-fp16-b8"),
        # int8 per channel with the opt-in fp16 recurrent state
        dict(_model_case("decode", "2.9B", "w8", "fp16", state="fp16", batch=64), name="decode-2.9B-w8-b64-s16"),
        # a server's step: 37 of 48 live requests scheduled, scattered over the slots
        dict(_model_case("serve", "2.9B", "w8", "fp16", capacity=48, batch=37), name="serve-2.9B-w8-37of48"),
        # bulk prefill, one chunk of 64 long prompts
        dict(_model_case("prefill", "7.2B", "mm4", "fp16", batch=64, tokens=512, scan_chunk=64), name="prefill-7.2B-mm4-64x512"),
        # a few prompts of no particular length through forward()
        dict(_model_case("prefill", "2.9B", "w8", "fp16", batch=3, tokens=777, scan_chunk=0), name="prefill-2.9B-w8-3x777"),
        # one prompt through the small model in fp32
        dict(_model_case("prefill", "0.1B", "dense", "fp32", batch=1, tokens=512, scan_chunk=0), name="prefill-0.1B-fp32-1x512"),
        # the recurrence alone over long sequences
        dict(kind="scan", batch=8, tokens=4096, heads=32, chunk=64, name="scan-8x4096x32"),
        # one int8 projection of a prompt chunk
        dict(kind="a8w8", rows=4096, k=4096, n=16384, name="a8w8-4096x4096x16384"),
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, round(math.exp(rng.uniform(math.log(lo), math.log(hi))))))


def draw(rng):
    kind = rng.choice(("decode", "decode", "decode", "serve", "prefill", "prefill", "scan", "a8w8"))
    if kind == "scan":
        heads, batch = rng.choice((12, 32, 40, 64)), rng.randint(1, 8)
        chunk = rng.choice((16, 32, 64))
        top = min(4096, 8 * 4096 * 32 // (heads * batch))
        return dict(kind="scan", batch=batch, tokens=chunk * _log_int(rng, 1, top // chunk), heads=heads, chunk=chunk)
    if kind == "a8w8":
        k, n = rng.choice(((2560, 2560), (2560, 10240), (10240, 2560), (4096, 4096), (4096, 16384), (16384, 4096)))
        return dict(kind="a8w8", rows=_log_int(rng, 64, 4096), k=k, n=n)
    shape = rng.choice(tuple(SHAPES))
    weights, dtype = rng.choice(FORMATS[shape])
    if kind == "decode":
        state = rng.choice(("fp32", "fp32", "fp16")) if dtype == "fp16" else "fp32"
        return _model_case(kind, shape, weights, dtype, state=state, batch=_log_int(rng, 1, 256))
    if kind == "serve":
        batch = _log_int(rng, 1, 96)
        return _model_case(kind, shape, weights, dtype, capacity=batch + rng.randint(0, 32), batch=batch)
    batch = _log_int(rng, 1, 64)
    tokens = _log_int(rng, 16, 2048)
    tokens = max(1, min(tokens, MAX_PREFILL // batch))
    if dtype == "fp16" and rng.random() < 0.5:
        return _model_case(kind, shape, weights, dtype, batch=batch, tokens=max(64, tokens // 64 * 64), scan_chunk=64)
    return _model_case(kind, shape, weights, dtype, batch=batch, tokens=tokens, scan_chunk=0)


# ------------------------------------------------------------------------------------------ states
def _build(case, gen):
    """A model of the case's shape with random weights: Linear ~ N(0, 0.02), the token-shift and key-scale parameters in
    the ranges of trained models, so that every term of the recurrence counts; projections quantised."""
    L, D, H, F = SHAPES[case["shape"]]
    cfg = hb.NativeRWKV7Config(vocab_size=VOCAB, hidden_size=D, num_hidden_layers=L, num_heads=H, head_dim=64,
                               intermediate_size=F, **RANKS)
    old = torch.get_default_dtype()
    torch.set_default_dtype(DTYPES[case["dtype"]])
    try:
        with torch.device(DEV):
            model = hb.RWKV7ForCausalLM(cfg, state_dtype=DTYPES[case.get("state", "fp32")]).eval()
    finally:
        torch.set_default_dtype(old)
    with torch.no_grad():
        for name, p in model.named_parameters():
            if p.dim() == 2:
                p.normal_(0.0, 1.0 if "embeddings" in name else 0.02, generator=gen)
        for i, layer in enumerate(model.model.layers):
            at = layer.attn
            for mix in (at.x_r, at.x_w, at.x_k, at.x_v, at.x_a, at.x_g, layer.ffn.x_k):
                mix.uniform_(0, 1, generator=gen)
            at.k_k.normal_(0.85, 0.1, generator=gen)
            at.k_a.normal_(1.0, 0.1, generator=gen)
            at.r_k.normal_(0.0, 0.1, generator=gen)
            at.w_lora.lora[2].bias.uniform_(-5, -1, generator=gen)
            at.a_lora.lora[2].bias.normal_(0, 0.5, generator=gen)
            if i:
                at.v_lora.lora[2].bias.normal_(0, 0.5, generator=gen)
    if case["weights"] != "dense":
        hb.quantize_model(model, case["weights"], min_params=1_000_000, group_size=128, skip=("lm_head",))
    return model


def _ids(gen, *shape):
    return torch.randint(0, VOCAB, shape, generator=gen, device=DEV)


def prepare(case, seed):
    gen = torch.Generator(device=DEV).manual_seed(int(seed))
    kind = case["kind"]
    if kind == "scan":
        B, T, H = case["batch"], case["tokens"], case["heads"]
        n = lambda: torch.randn(B, T, H, 64, generator=gen, device=DEV)
        r, k, v = n().half(), n().half(), n().half()
        kk = torch.nn.functional.normalize(k.float(), dim=-1).half()
        return dict(case=case, args=(r, torch.exp(-0.606531 * torch.sigmoid(n())), k, v, kk, torch.sigmoid(n()).half(),
                                     torch.zeros(B, H, 64, 64, device=DEV)))
    if kind == "a8w8":
        lin = torch.nn.Linear(case["k"], case["n"], bias=False, device=DEV, dtype=torch.float16)
        with torch.no_grad():
            lin.weight.normal_(0.0, 0.02, generator=gen)
        x = torch.randn(case["rows"], case["k"], generator=gen, device=DEV).half()
        return dict(case=case, linear=hb.A8W8Linear(lin), x=x)
    model = _build(case, gen)
    B = case["batch"]
    state = dict(case=case, model=model)
    if kind == "prefill":
        state["ids"] = _ids(gen, B, case["tokens"])
        return state
    prompt, state["ids"] = _ids(gen, B, PROMPT), _ids(gen, B)
    if kind == "decode":
        # the program has prefilled its prompts and produced one token (which captured the step's graph)
        _, cache = model.rwkv7_prefill_native(prompt)
        model.rwkv7_forward_token(_ids(gen, B), cache)
        state["cache"] = cache
        return state
    pool = hb.RWKV7StatePool(model, case["capacity"])
    slots, generations = pool.allocate(range(case["capacity"]))
    order = torch.randperm(case["capacity"], generator=gen, device=DEV).tolist()[:B]
    state.update(pool=pool, slots=[slots[i] for i in order], generations=[generations[i] for i in order])
    pool.prefill(prompt, state["slots"], state["generations"])
    pool.decode(_ids(gen, B), state["slots"], state["generations"])
    return state


def _cache_outputs(logits, cache):
    """Logits and the updated cache.  The shift states come from the last layers only, which depend on all before them:
    a checker takes no more than 64 tensors."""
    state, xpa, xpf, v_first = cache
    tail = min(len(state), (64 - 2 - len(state)) // 2)
    return dict(logits=logits, state=list(state), v_first=v_first, xpa=list(xpa[-tail:]), xpf=list(xpf[-tail:]))


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "decode":
        return _cache_outputs(state["model"].rwkv7_forward_token(state["ids"], state["cache"]), state["cache"])
    if kind == "serve":
        pool = state["pool"]
        logits = pool.decode(state["ids"], state["slots"], state["generations"])
        n = pool.capacity  # the row behind the slots is the padding rows' scratch: no request's state
        return dict(logits=logits, state=pool.S_pool[:, :n], xpa=pool.xpa_pool[:, :n], xpf=pool.xpf_pool[:, :n],
                    v_first=pool.vfirst_pool[:n])
    if kind == "prefill":
        if case["scan_chunk"]:
            logits, cache = state["model"].rwkv7_prefill_chunks(state["ids"], chunk_size=512, scan_chunk=case["scan_chunk"])
        else:
            out = state["model"](input_ids=state["ids"], logits_to_keep=1)
            logits, cache = out.logits, out.past_key_values
        return _cache_outputs(logits, cache)
    if kind == "scan":
        return hb.self_chunk_rwkv7(*state["args"], chunk_size=case["chunk"])
    return state["linear"](state["x"])


# ------------------------------------------------------------------------------------------ what a pass needs
def work(case):
    """Bytes that have to move once and operations (two per multiply-add) of one pass."""
    kind = case["kind"]
    if kind == "scan":
        th, bh = case["batch"] * case["tokens"] * case["heads"], case["batch"] * case["heads"]
        # r, k, v, kk, a, y in fp16 and w in fp32; state in and out.  Per token and head: decay, S.a, two rank-one terms, S.r
        return {"bytes": th * 64 * (6 * 2 + 4) + 2 * bh * 4096 * 4, "flops": th * 4096 * 9}
    if kind == "a8w8":
        M, K, N = case["rows"], case["k"], case["n"]
        return {"bytes": M * K * 2 + K * N + N * 4 + M * N * 2, "flops": 2 * M * K * N}
    L, D, H, F = SHAPES[case["shape"]]
    B, T = case["batch"], case.get("tokens", 1)
    e = 4 if case["dtype"] == "fp32" else 2
    proj = 4 * D * D + 2 * D * F
    lora = 2 * D * sum(RANKS.values())
    weights = {"dense": proj * e, "w8": proj + (4 * D + 2 * F) * 2, "mm4": proj // 2 + proj // 128 * 2}[case["weights"]]
    state = L * H * 4096 * (2 if case.get("state") == "fp16" else 4) + 2 * L * D * e
    reads = 1 if kind == "prefill" else 2  # a prefill starts from the zero state
    bytes_ = L * (weights + lora * e) + VOCAB * D * e + B * (reads * state + VOCAB * e) + B * T * (8 + D * e)
    flops = 2 * B * T * L * (proj + lora) + 2 * B * VOCAB * D + B * T * L * H * 4096 * 9
    return {"bytes": bytes_, "flops": flops}


def tolerance(case):
    """About four times the difference that was measured against the same path with its sums in another order: the
    projections of a model through other kernels (weights streamed or dequantised first, K in two halves), the scan
    token by token, the int8 projection in 64 bits."""
    if case["kind"] == "scan":
        return {"rel": 2e-3, "max": 2e-2}  # measured 4.6e-4 / 4.2e-3
    if case["kind"] == "a8w8":
        return {"rel": 8e-4, "max": 2e-3}  # measured 2.1e-4 / 4.9e-4: the rounding of the result alone
    return {"fp32": {"rel": 6e-6, "max": 5e-5},  # measured 1.5e-6 / 1.2e-5
            "fp16": {"rel": 1.2e-2, "max": 0.2},  # measured 3.2e-3 / 4.4e-2 (the state after 32 layers is the furthest)
            "bf16": {"rel": 3e-2, "max": 0.5}}[case["dtype"]]
