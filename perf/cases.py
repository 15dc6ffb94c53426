"""What a user of this package has it do, as a list of cases that can be timed.

Four kinds of work, each through the public call that a user makes:

  attention   custom_flash_attn.forward on q, k, v of [B, H, N, 64]: the drop-in call itself
  decode      custom_flash_attn.decode: one new token per sequence against a K/V cache
  generate    gpt2.generate: prompt, then token by token (greedy); by default arguments, or with the
              GenerationSession that a program with many prompts keeps
  steps       the single-token step of a GenerationSession for a batch that already has its prompt
              in the cache, the next tokens given (a server's decode loop, or scoring a continuation)
  prefill     GPTModel over whole sequences, logits of every position (GPTModel.capture_prefill)

Head dimension 64 and bf16 are what the attention kernels take.  Models are the GPT-2 sizes of
gpt2.GPT2_SIZES in bf16 with random weights, prepared for inference.
"""
import math

import torch

from tfg_flashattention_b200 import custom_flash_attn, gpt2

D = 64
VOCAB = 50257
CONTEXT = 1024


def listed():
    return [
        # the shortest call: one 72-token prompt, one GPT-2 small layer; the host's time and the launch
        dict(name="attn_prompt", kind="attention", B=1, H=12, N=72, causal=True, lse=False, layout="bhnd"),
        # GPT-2 small, four full sequences: less than two tiles of work per resident block
        dict(name="attn_small", kind="attention", B=4, H=12, N=1024, causal=True, lse=False, layout="bhnd"),
        # odd length, read in place from a fused QKV projection as the GPT-2 module does, LSE asked for
        dict(name="attn_ragged_lse", kind="attention", B=8, H=16, N=777, causal=True, lse=True, layout="qkv"),
        # one GPT-2 XL layer at batch 32: the benchmark's headline shape
        dict(name="attn_xl_layer", kind="attention", B=32, H=25, N=1024, causal=True, lse=False, layout="bhnd"),
        # unmasked attention, long enough that the tile loop is all there is
        dict(name="attn_full", kind="attention", B=16, H=16, N=4096, causal=False, lse=True, layout="bhnd"),
        # long context, causal
        dict(name="attn_long", kind="attention", B=4, H=25, N=16384, causal=True, lse=False, layout="bhnd"),
        # one sequence's step: latency of a single call
        dict(name="decode_one", kind="decode", B=1, H=25, kv_len=900, rows=1024, append=True, lse=False, layout="bnhd"),
        # a batch's step over the model's own cache layout, lengths that are no round number
        dict(name="decode_batch", kind="decode", B=32, H=25, kv_len=1001, rows=1024, append=True, lse=False,
             layout="bnhd"),
        # a long cache, as the attention call alone would meet it
        dict(name="decode_long", kind="decode", B=8, H=25, kv_len=8192, rows=8192, append=False, lse=True,
             layout="bhnd"),
        # 72 tokens of prompt and 20 new ones, GPT-2 small, one sequence, default arguments
        dict(name="generate_small", kind="generate", model="gpt2-small", B=1, prompt=72, new=20, session=False),
        # eight sequences of GPT-2 XL, 24 steps behind a 900-token prompt
        dict(name="steps_xl", kind="steps", model="gpt2-xl", B=8, prompt=900, new=24),
        # GPT-2 small over 8 x 1024 tokens, all logits
        dict(name="prefill_small", kind="prefill", model="gpt2-small", B=8, N=1024),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    most = max(_cost(c) for c in listed())
    while True:
        kind = rng.choice(["attention"] * 6 + ["decode"] * 3 + ["generate", "steps", "prefill"])
        if kind == "attention":
            c = dict(kind=kind, B=_log_int(rng, 1, 32), H=rng.choice([12, 16, 20, 25]), N=_log_int(rng, 16, 16384),
                     causal=rng.random() < 0.75, lse=rng.random() < 0.4, layout=rng.choice(["bhnd", "qkv"]))
            # no more than the largest attention problem of the list
            if (1 if c["causal"] else 2) * c["B"] * c["H"] * c["N"] ** 2 > 4 * 25 * 16384 ** 2:
                continue
        elif kind == "decode":
            kv = _log_int(rng, 32, 16384)
            c = dict(kind=kind, B=_log_int(rng, 1, 64), H=rng.choice([12, 16, 20, 25]), kv_len=kv,
                     rows=max(kv, 1024), append=rng.random() < 0.6, lse=rng.random() < 0.4,
                     layout=rng.choice(["bnhd", "bhnd"]))
            if c["B"] * c["H"] * kv > 4 * 25 * 32768:
                continue
        elif kind == "generate":
            session = rng.random() < 0.5
            c = dict(kind=kind, model=rng.choice(sorted(gpt2.GPT2_SIZES)), B=rng.choice([1, 1, 2, 4]),
                     prompt=_log_int(rng, 8, 512), new=rng.randint(4, 20 if session else 8), session=session)
        elif kind == "steps":
            c = dict(kind=kind, model=rng.choice(sorted(gpt2.GPT2_SIZES)), B=_log_int(rng, 1, 8),
                     prompt=_log_int(rng, 16, 960), new=rng.randint(4, 20))
        else:
            c = dict(kind=kind, model=rng.choice(["gpt2-small", "gpt2-medium"]), B=_log_int(rng, 1, 8),
                     N=_log_int(rng, 64, 1024))
        if _cost(c) <= most:
            return c


# ---------------------------------------------------------------------------------- inputs

def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _normal(g, *shape):
    return torch.randn(*shape, device="cuda", generator=g, dtype=torch.bfloat16)


def _model(name, seed):
    """GPT-2 of the named size in bf16 with seeded weights: N(0, 0.02), the two projections that write
    to the residual stream scaled by 1/sqrt(2 * layers) as GPT-2 initialises them, token embeddings
    with a trained model's spread (0.14).  Each row of the output head also carries the direction of
    one token's embedding (a seeded permutation says whose), so the model is sure of its next token
    by far more than the rounding of another correct implementation could move, as a trained model
    decoding greedily mostly is, and token ids can be compared."""
    cfg = gpt2.gpt2_config(name, impl_type="cuda", context_length=CONTEXT)
    with torch.device("cuda"):
        model = gpt2.GPTModel(cfg, dtype=torch.bfloat16).eval()
    g = _generator(seed)
    with torch.no_grad():
        for key, prm in model.named_parameters():
            if key.endswith(".scale"):
                prm.fill_(1.0)
            elif key.endswith(".shift"):
                prm.zero_()
            else:
                std = 0.02
                if key.endswith(("out_proj.weight", "layers.2.weight")):
                    std /= math.sqrt(2.0 * cfg["n_layers"])
                elif key.startswith("tok_emb"):
                    std = 0.14
                prm.normal_(0.0, std, generator=g)
        follows = torch.randperm(VOCAB, device="cuda", generator=g)
        emb = model.tok_emb.weight.float()
        model.out_head.weight[follows] += (2.0 * emb / emb.norm(dim=1, keepdim=True)).bfloat16()
    return model.prepare_for_inference()


def _ids(g, *shape):
    return torch.randint(0, VOCAB, shape, device="cuda", generator=g)


def prepare(case, seed):
    kind = case["kind"]
    g = _generator(seed)
    state = dict(case)
    if kind == "attention":
        B, H, N = case["B"], case["H"], case["N"]
        if case["layout"] == "qkv":      # column slices of one [B, N, 3, H, 64] projection
            qkv = _normal(g, B, N, 3, H, D)
            state["q"], state["k"], state["v"] = (qkv[:, :, i].transpose(1, 2) for i in range(3))
        else:
            state["q"], state["k"], state["v"] = (_normal(g, B, H, N, D) for _ in range(3))
    elif kind == "decode":
        B, H, rows = case["B"], case["H"], case["rows"]
        if case["layout"] == "bnhd":     # GPTModel.allocate_kv_cache's layout
            state["k"], state["v"] = (_normal(g, B, rows, H, D).transpose(1, 2) for _ in range(2))
        else:
            state["k"], state["v"] = (_normal(g, B, H, rows, D) for _ in range(2))
        qkv = _normal(g, B, 1, 3, H, D)
        state["q"], state["k_new"], state["v_new"] = (qkv[:, :, i].transpose(1, 2) for i in range(3))
    elif kind == "prefill":
        model = _model(case["model"], seed)
        state["ids"] = _ids(g, case["B"], case["N"])
        state["forward"] = model.capture_prefill(case["B"], case["N"])
        state["model"] = model
    else:
        model = _model(case["model"], seed)
        state["ids"] = _ids(g, case["B"], case["prompt"])
        state["gpt"] = model
        if kind == "steps" or case["session"]:
            state["kept"] = gpt2.GenerationSession(model, case["B"], CONTEXT)
        if kind == "steps":
            with torch.no_grad():
                model(state["ids"], last_token_only=True, kv_caches=state["kept"].caches, pos=0)
            state["next"] = _ids(g, case["B"], case["new"])
    return state


# ---------------------------------------------------------------------------------- one pass

def run(state):
    kind = state["kind"]
    if kind == "attention":
        return custom_flash_attn.forward(state["q"], state["k"], state["v"], causal=state["causal"],
                                         return_lse=state["lse"])
    if kind == "decode":
        new = dict(k_new=state["k_new"], v_new=state["v_new"]) if state["append"] else {}
        out = custom_flash_attn.decode(state["q"], state["k"], state["v"], state["kv_len"],
                                       return_lse=state["lse"], **new)
        return (out, state["k"], state["v"]) if state["append"] else out
    if kind == "prefill":
        return state["forward"](state["ids"])
    if kind == "generate":
        return gpt2.generate(state["gpt"], state["ids"], state["new"], CONTEXT, temperature=0.0,
                             session=state.get("kept"))
    session, ids = state["kept"], state["next"]
    session.position.set(state["prompt"])
    # the step's logits live in the session and the next step overwrites them
    return [session.step_fn(ids[:, t:t + 1]).clone() for t in range(state["new"])]


# ---------------------------------------------------------------------------------- what it takes

def _model_work(name, rows, heads_rows):
    """Bytes of one pass over the weights, and operations for `rows` tokens of which `heads_rows`
    get logits (attention not included)."""
    size = gpt2.GPT2_SIZES[name]
    layers, width = size["n_layers"], size["emb_dim"]
    block, head = 12 * width * width, VOCAB * width
    return 2.0 * (layers * block + head), 2.0 * (rows * layers * block + heads_rows * head)


def work(case):
    kind = case["kind"]
    if kind == "attention":
        B, H, N = case["B"], case["H"], case["N"]
        return {"bytes": 8.0 * B * H * N * D + (4.0 * B * H * N if case["lse"] else 0.0),
                "flops": (2.0 * B * H * N * (N + 1) if case["causal"] else 4.0 * B * H * N * N) * D}
    if kind == "decode":
        B, H, kv = case["B"], case["H"], case["kv_len"]
        return {"bytes": 4.0 * B * H * kv * D + 4.0 * B * H * D + (4.0 * B * H * D if case["append"] else 0.0)
                + (4.0 * B * H if case["lse"] else 0.0),
                "flops": 4.0 * B * H * kv * D}
    layers, width = gpt2.GPT2_SIZES[case["model"]]["n_layers"], gpt2.GPT2_SIZES[case["model"]]["emb_dim"]
    B = case["B"]
    if kind == "prefill":
        N = case["N"]
        weights, flops = _model_work(case["model"], B * N, B * N)
        return {"bytes": weights + 2.0 * B * N * VOCAB, "flops": flops + 2.0 * B * N * (N + 1) * width * layers}
    total, flops = 0.0, 0.0
    n = case["prompt"]
    steps = case["new"]
    if kind == "generate":               # the prompt gives the first new token, a step each of the others
        weights, ops = _model_work(case["model"], B * n, B)
        total += weights + 4.0 * B * n * width * layers
        flops += ops + 2.0 * B * n * (n + 1) * width * layers
        steps -= 1
    weights, ops = _model_work(case["model"], B, B)
    for t in range(steps):
        total += weights + 4.0 * B * (n + t + 1) * width * layers + (2.0 * B * VOCAB if kind == "steps" else 0.0)
        flops += ops + 4.0 * B * (n + t + 1) * width * layers
    return {"bytes": total, "flops": flops}


def _cost(case):
    w = work(case)
    return max(w["bytes"], w["flops"] / 50)


def tolerance(case):
    kind = case["kind"]
    if kind == "generate":
        return "exact"                   # token ids
    if kind in ("attention", "decode"):
        # P and O are rounded to bf16: 2^-9 relative each, and the sums' order
        return {"rel": 1e-2, "max": 0.1}
    # dozens of bf16 roundings in a row, each of which another order of summation may flip
    return {"rel": 2e-2}
