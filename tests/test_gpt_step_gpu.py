"""The one-launch generation step (fa_b200_gpt_step, csrc/gpt_step_sm100.cuh) against the same model
evaluated in fp32 with the reference's standard-PyTorch attention.

Tolerance: the kernel rounds activations to bf16 about eight times per layer (LayerNorm outputs, q,
k, v, attention output, hidden row, and the stream where it is normalised) and the logits once.  Each
rounding (8 significant bits) adds at most 2^-8 of the value it rounds; treated as independent, the
relative error of the logits (2-norm) stays below 2^-8 * sqrt(8 L + 4)."""
import math

import pytest
import torch

from tfg_flashattention_b200 import gpt2

pytestmark = pytest.mark.gpu


def _model(width, heads, layers, vocab, context, qkv_bias=True, seed=3):
    cfg = {"vocab_size": vocab, "context_length": context, "emb_dim": width, "n_heads": heads, "n_layers": layers,
           "drop_rate": 0.0, "qkv_bias": qkv_bias, "impl_type": "cuda"}
    torch.manual_seed(seed)
    model = gpt2.GPTModel(cfg, dtype=torch.bfloat16)
    with torch.no_grad():
        for name, p in model.named_parameters():
            if name.endswith(".scale"):
                p.copy_(1 + 0.2 * torch.randn(p.shape))
            elif name.endswith("emb.weight"):
                p.copy_(torch.randn(p.shape))
            elif p.dim() == 2:
                p.copy_(torch.randn(p.shape) / math.sqrt(p.shape[1]))
            else:
                p.copy_(0.3 * torch.randn(p.shape))
    exact = gpt2.GPTModel(dict(cfg, impl_type="manual"))
    exact.load_state_dict(model.state_dict())
    model = model.cuda().eval().prepare_for_inference()
    assert model._step_plan is not None
    return model, exact.cuda().eval()


def _check(model, exact, B, pos, seed=0, **kw):
    """One step at position `pos` behind `pos` cached rows of the exact model (rounded to bf16)."""
    cfg = model.cfg
    ids = torch.randint(0, cfg["vocab_size"], (B, pos + 1), generator=torch.Generator().manual_seed(seed)).cuda()
    caches = model.allocate_kv_cache(B, pos + 2)
    wide = [tuple(t.float() for t in pair) for pair in caches]
    with torch.no_grad():
        if pos:
            exact(ids[:, :pos], kv_caches=wide, pos=0)
            for (k, v), (kw_, vw) in zip(caches, wide):
                k.copy_(kw_)
                v.copy_(vw)
                kw_.copy_(k)
                vw.copy_(v)
        want = exact(ids[:, pos:], kv_caches=wide, pos=pos)
        before = [tuple(t.clone() for t in pair) for pair in caches]
        nxt = torch.full((B, 3), -1, dtype=torch.long, device="cuda")
        got = model._step(ids[:, pos:], caches, pos, next_ids=nxt[:, 1])
    from tfg_flashattention_b200 import custom_flash_attn
    assert custom_flash_attn.last_status() == 0
    assert got is not None and got.shape == want.shape
    L = cfg["n_layers"]
    bound = 2.0 ** -8 * math.sqrt(8 * L + 4)
    rel = ((got.float() - want).norm() / want.norm()).item()
    assert rel <= bound, (rel, bound)
    # the argmax is that of the logits themselves; the columns beside it are not touched
    assert torch.equal(nxt[:, 1], got[:, 0].float().argmax(-1)) and (nxt[:, ::2] == -1).all()
    for (k, v), (kw_, vw), (k0, v0) in zip(caches, wide, before):
        for new, ref, old in ((k, kw_, k0), (v, vw, v0)):
            assert ((new[:, pos].float() - ref[:, pos]).norm() / ref[:, pos].norm()).item() <= bound
            keep = torch.arange(new.shape[1], device="cuda") != pos
            assert torch.equal(new[:, keep], old[:, keep])               # nothing else is written
    return caches, ids, got


@pytest.mark.parametrize("width,heads,layers,vocab,B,pos,bias", [
    (64, 1, 2, 97, 1, 0, True),          # no cached rows; fewer rows of W than CTAs
    (64, 1, 1, 97, 8, 1, True),
    (320, 5, 2, 503, 3, 15, False),      # 10 columns units: warps without work; no QKV bias
    (768, 12, 2, 1001, 1, 16, True),     # one chunk per row
    (768, 12, 1, 1001, 5, 95, True),     # cached rows: one stage less one, ...
    (1024, 16, 1, 1001, 2, 96, True),    # ... exactly one, ...
    (1280, 20, 1, 1001, 4, 97, True),    # ... and one row into the second
    (1600, 25, 2, 50257, 8, 130, True),  # two attention units in some CTAs; the widest model
])
def test_step_matches_fp32(fa_lib, width, heads, layers, vocab, B, pos, bias):
    _check(*_model(width, heads, layers, vocab, 256, bias), B, pos)


@pytest.mark.parametrize("B,heads,pos", [(1, 1, 2047), (1, 1, 2048), (2, 2, 5000),     # pairs in parts, more than 8 of them
                                         (1, 12, 767), (1, 12, 768),       # the border: one CTA a pair, two
                                         (1, 12, 272), (1, 12, 289),       # a pair a CTA: whole blocks of 16 rows, one more
                                         (8, 25, 193), (8, 25, 901),       # 200 pairs: two in some CTAs
                                         (8, 12, 900), (5, 16, 480)])      # fewer pairs than CTAs, not enough to split
def test_step_long_cache_is_split_over_ctas(fa_lib, B, heads, pos):
    _check(*_model(64 * heads, heads, 1, 211, pos + 8), B, pos)


def test_step_advances_a_device_position_and_repeats_bit_for_bit(fa_lib):
    model, exact = _model(256, 4, 2, 503, 64)
    caches, ids, first = _check(model, exact, 2, 20)
    position = gpt2.DevicePosition(torch.device("cuda", torch.cuda.current_device()))
    position.set(20)
    for _ in range(3):
        position.set(20)
        again = model._step(ids[:, 20:], caches, position, advance=True)
        assert torch.equal(again, first)
        assert position.index.item() == 21 and position.length.item() == 22
    # a replaced parameter is seen: the table is rebuilt
    model.trf_blocks[0].ff.layers[0].bias = torch.nn.Parameter(model.trf_blocks[0].ff.layers[0].bias + 1)
    assert not torch.equal(model._step(ids[:, 20:], caches, 20), first)


def test_step_declines_what_it_does_not_take(fa_lib):
    model, _ = _model(256, 4, 1, 503, 64)
    ids = torch.zeros(2, 1, dtype=torch.long, device="cuda")
    caches = model.allocate_kv_cache(2, 32)
    assert model._step(ids, caches, 31) is not None
    assert model._step(ids, caches, 32) is None                              # past the cache
    assert model._step(ids, model.allocate_kv_cache(2, 32, dtype=torch.float32), 3) is None
    assert model._step(torch.zeros(9, 1, dtype=torch.long, device="cuda"), model.allocate_kv_cache(9, 32), 3) is None


@pytest.mark.parametrize("lose", ["to", "invalidate", "prepare"])
def test_recorded_step_keeps_what_it_reads(fa_lib, lose):
    """The graph holds the address of the parameter table, the table those of the weights.  (Whether they
    are still owned is looked at before anything is replayed.)"""
    import gc
    model, exact = _model(256, 4, 2, 503, 64)
    session = gpt2.GenerationSession(model, 2, 64)
    read = [model._step_plan.table] + [w for _, w, *_ in model._step_plan.qkv]
    addresses = [t.untyped_storage().data_ptr() for t in read]
    del read
    ids = torch.randint(0, 503, (2, 1), device="cuda")
    session.position.set(0)
    before = session.step_fn(ids).clone()
    {"to": lambda: model.to("cuda"), "invalidate": model.invalidate_inference_cache, "prepare": model.prepare_for_inference}[lose]()
    gc.collect()
    torch.cuda.synchronize()
    taken = [torch.full((n,), 7, dtype=torch.uint8, device="cuda") for n in (512, 1024, 2048, 400000) for _ in range(8)]
    kept = {t.untyped_storage().data_ptr() for t in getattr(session.step_fn, "reads", []) if isinstance(t, torch.Tensor)}
    assert kept.issuperset(addresses) and len(taken) == 32
    session.position.set(0)
    assert torch.equal(session.step_fn(ids), before)


def test_graph_of_the_caller_keeps_the_table(fa_lib):
    """The same for a graph that a program records around the model itself; the weights stay in place."""
    import gc
    model, exact = _model(256, 4, 2, 503, 64)
    caches = model.allocate_kv_cache(2, 64)
    ids = torch.randint(0, 503, (2, 1), device="cuda")
    with torch.no_grad():
        before = model(ids, kv_caches=caches, pos=5)
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            out = model(ids, kv_caches=caches, pos=5)
    weights, table = [w for _, w, *_ in model._step_plan.qkv], model._step_plan.table.data_ptr()
    model.invalidate_inference_cache()
    gc.collect()
    assert [t.data_ptr() for t in getattr(model, "_recorded_tables", [])] == [table] and len(weights) == 2
    out.zero_()
    graph.replay()
    assert torch.equal(out, before)


@pytest.mark.parametrize("B", [8, 9, 11])
def test_session_of_more_sequences_than_the_kernel_takes(fa_lib, B):
    """... is recorded layer by layer, and generates what the same sequences give in two sessions."""
    model, _ = _model(256, 4, 2, 503, 64)
    ids = torch.randint(0, 503, (B, 5), generator=torch.Generator().manual_seed(B)).cuda()
    session = gpt2.GenerationSession(model, B, 64)
    assert (session.step_fn.workspace is not None) == (B <= 8)
    step, position, caches = session.step_fn, session.position, session.caches
    with torch.no_grad():
        model(ids[:, :4], kv_caches=caches, pos=0)
        position.set(4)
        got = step(ids[:, 4:]).float()
        parts = []
        for half in ids.split(4):
            part = model.allocate_kv_cache(half.shape[0], 64)
            model(half[:, :4], kv_caches=part, pos=0)
            parts.append(model(half[:, 4:], kv_caches=part, pos=4).float())
    want = torch.cat(parts)
    # two layers at the tolerance of the file's head, each side with its own roundings
    assert ((got - want).norm() / want.norm()).item() <= 2 * 2.0 ** -8 * math.sqrt(8 * 2 + 4)
    out = gpt2.generate(model, ids, 4, 64, temperature=0.0, session=session)
    assert out.shape == (B, 9) and torch.equal(out[:, :5], ids)


@pytest.mark.parametrize("B", [1, 2])
@pytest.mark.parametrize("where", ["tok_emb", "att", "ff", "out_proj", "layers.2", "forward", "autocast"])
def test_step_leaves_calls_to_the_modules(fa_lib, where, B):
    """Hooks and a module's own forward are called as often as the layer-by-layer loop calls them, in steps and
    in prompts; under autocast nothing goes past the modules."""
    model, _ = _model(256, 4, 2, 503, 64)
    blk = model.trf_blocks[1]
    module = {"tok_emb": model.tok_emb, "att": blk.att, "ff": blk.ff, "out_proj": blk.att.out_proj,
              "layers.2": blk.ff.layers[2], "forward": blk.att, "autocast": blk.att}[where]
    ids = torch.randint(0, 503, (B, 6), device="cuda")

    def run():
        seen = []
        caches = model.allocate_kv_cache(B, 32)
        if where == "forward":
            inner = type(module).forward
            module.forward = lambda *a, **k: (seen.append(1), inner(module, *a, **k))[1]
        elif where != "autocast":
            handle = module.register_forward_hook(lambda *a: seen.append(1))
        with torch.no_grad(), torch.autocast("cuda", dtype=torch.bfloat16, enabled=where == "autocast"):
            model(ids[:, :5], kv_caches=caches, pos=0)
            prompt = len(seen)
            taken = model._step(ids[:, 5:], caches, 5)
            out = model(ids[:, 5:], kv_caches=caches, pos=5).float()
        if where == "forward":
            del module.forward
        elif where != "autocast":
            handle.remove()
        return prompt, len(seen) - prompt, taken, out

    prompt, step, taken, out = run()
    assert taken is None
    model._native_blocks, model._step = lambda *a: None, lambda *a, **k: None
    want = run()
    assert (prompt, step) == want[:2] and torch.equal(out, want[3])
    del model._native_blocks, model._step
    assert model._step(ids[:, 5:], model.allocate_kv_cache(B, 32), 5) is not None


@pytest.mark.parametrize("new", [1, 4])
def test_session_goes_on_behind_what_was_generated(fa_lib, new):
    """generate() leaves the session's position behind its last step, greedy or sampled, so that the recorded
    step can go on."""
    model, _ = _model(256, 4, 2, 503, 64)
    ids = torch.randint(0, 503, (2, 7), device="cuda")
    for temperature in (0.0, 1.0):
        session = gpt2.GenerationSession(model, 2, 64)
        out = gpt2.generate(model, ids, new, 64, temperature=temperature, session=session)
        assert session.position.index.item() == 7 + new - 1 and session.position.length.item() == 7 + new
        got = session.step_fn(out[:, -1:]).clone()
        caches = model.allocate_kv_cache(2, 64)
        with torch.no_grad():
            model(out[:, :7], kv_caches=caches, pos=0)
            for t in range(7, 7 + new):
                want = model(out[:, t:t + 1], kv_caches=caches, pos=t)
        assert torch.equal(got, want)


@pytest.mark.parametrize("how", ["hook", "pre-hook", "forward", "subclass"])
def test_generate_calls_the_model_where_somebody_waits_for_it(fa_lib, how):
    model, _ = _model(256, 4, 2, 503, 64)
    ids = torch.randint(0, 503, (2, 7), device="cuda")
    want = gpt2.generate(model, ids, 5, 64, temperature=0.0)
    seen = []
    if how == "hook":
        model.register_forward_hook(lambda *a: seen.append(1))
    elif how == "pre-hook":
        model.register_forward_pre_hook(lambda *a: seen.append(1))
    elif how == "forward":
        model.forward = lambda *a, **k: (seen.append(1), gpt2.GPTModel.forward(model, *a, **k))[1]
    else:
        class Model(gpt2.GPTModel):
            def forward(self, *a, **k):
                seen.append(1)
                return super().forward(*a, **k)
        model.__class__ = Model
    assert torch.equal(gpt2.generate(model, ids, 5, 64, temperature=0.0), want) and len(seen) == 5


def test_positions_of_other_integer_types(fa_lib):
    import numpy as np
    model, _ = _model(256, 4, 2, 503, 64)
    ids = torch.randint(0, 503, (2, 7), device="cuda")
    caches = model.allocate_kv_cache(2, 32)
    with torch.no_grad():
        model(ids[:, :6], kv_caches=caches, pos=np.int64(0))
        want = model(ids[:, 6:], kv_caches=caches, pos=6)
        for kind in (np.int64, np.int32, np.uint8):
            assert torch.equal(model(ids[:, 6:], kv_caches=caches, pos=kind(6)), want)


@pytest.mark.parametrize("generation", [65530, 65534, 0xfffffffb, 0xffffffff])
def test_steps_across_the_wrap_of_the_generation(fa_lib, generation):
    """The exchange words carry 16 bits of a counter that goes up by layers + 1 a step.  Steps from a counter
    shortly before it wraps (in 16 bits, and in the 32 it is kept in) against a fresh workspace's, to the bit."""
    model, _ = _model(768, 12, 2, 503, 64)
    plan = model._step_plan
    ids = torch.randint(0, 503, (4, 12), device="cuda")
    runs = []
    for start in (0, generation):
        caches = model.allocate_kv_cache(4, 16)
        workspace = plan.new_workspace(4)
        outs = [model._step(ids[:, t:t + 1], caches, t, workspace=workspace) for t in range(3)]
        if start:
            workspace.view(torch.int32)[0] = start - (start >> 31 << 32)
        outs += [model._step(ids[:, t:t + 1], caches, t, workspace=workspace) for t in range(3, 12)]
        runs.append((torch.cat(outs), [torch.cat(pair) for pair in caches]))
    assert torch.equal(runs[0][0], runs[1][0])
    assert all(torch.equal(a, b) for a, b in zip(runs[0][1], runs[1][1]))


def test_head_strides_past_32_bits(fa_lib):
    """Caches whose last head lies more than 2^31 elements behind the first (one allocation of 4.5 GB, K and V
    interleaved in it): the new row goes where it belongs and nowhere else."""
    model, _ = _model(1600, 25, 1, 503, 64)
    stride = 2 ** 31 // 24 // 8 * 8 + 64
    flat = torch.zeros(24 * stride + 4096, dtype=torch.bfloat16, device="cuda")
    wide = [tuple(flat[at:].as_strided((1, 16, 25, 64), (64, 64, stride, 1)) for at in (0, 2048))]
    assert wide[0][0].stride(2) * 24 > 2 ** 31
    caches = model.allocate_kv_cache(1, 16)
    ids = torch.randint(0, 503, (1, 6), device="cuda")
    with torch.no_grad():
        for t in range(6):
            want = model._step(ids[:, t:t + 1], caches, t)
            got = model._step(ids[:, t:t + 1], wide, t)
            assert torch.equal(got, want)
    for a, b in zip(caches[0], wide[0]):
        assert torch.equal(a, b)
    assert int((flat != 0).sum()) == sum(int((t != 0).sum()) for t in caches[0])


@pytest.mark.parametrize("B,pos", [(1, 0), (2, 5), (1, 200)])
def test_scores_far_below_zero(fa_lib, B, pos):
    """A layer whose scores are all about -1e33 against the same model layer by layer."""
    model, _ = _model(256, 4, 1, 503, 256)
    att = model.trf_blocks[0].att
    with torch.no_grad():
        att.W_query.weight.zero_()
        att.W_key.weight.zero_()
        att.W_query.bias.fill_(1e16)
        att.W_key.bias.fill_(-1e16)
    model.prepare_for_inference()
    ids = torch.randint(0, 503, (B, pos + 1), generator=torch.Generator().manual_seed(1)).cuda()
    runs = []
    with torch.no_grad():
        for stepped in (True, False):
            caches = model.allocate_kv_cache(B, 256)
            if pos:
                model(ids[:, :pos], kv_caches=caches, pos=0)
            if not stepped:
                model._step = lambda *a, **k: None
            runs.append(model(ids[:, pos:], kv_caches=caches, pos=pos).float())
    got, want = runs
    assert torch.isfinite(got).all()
    assert ((got - want).norm() / want.norm()).item() <= 2 * 2.0 ** -8 * math.sqrt(8 + 4)


@pytest.mark.parametrize("heads,B", [(25, 1), (25, 8), (12, 1), (12, 3), (1, 2)])
@pytest.mark.parametrize("row", ["far from 0", "outlier in front", "outlier behind"])
def test_layernorm_of_ill_conditioned_rows(fa_lib, heads, B, row):
    """The first LayerNorm's output, taken from the K cache behind an identity projection, against fp64.  It is
    rounded to bf16 twice (2^-9 each, as LayerNorm's output and as K, whose products with 1 and 0 are exact);
    the variance may lose C * 2^-24 * 2 (see step_layernorm), half of that in the result."""
    C = 64 * heads
    model, _ = _model(C, heads, 1, 97, 64)
    g = torch.Generator().manual_seed(heads)
    flip = torch.randint(0, 2, (97, C), generator=g).float()
    if row == "far from 0":
        emb = 448 + 2 * flip                             # neighbours in bf16
    else:
        emb = (flip - 0.5) / 16
        emb[:, 0 if row == "outlier in front" else C - 1] = 200.0
    with torch.no_grad():
        model.tok_emb.weight.copy_(emb)
        model.pos_emb.weight.zero_()
        blk = model.trf_blocks[0]
        blk.att.W_key.weight.copy_(torch.eye(C))
        blk.att.W_key.bias.zero_()
        blk.norm1.scale.fill_(1)
        blk.norm1.shift.zero_()
    model.prepare_for_inference()
    caches = model.allocate_kv_cache(B, 8)
    ids = torch.randint(0, 97, (B, 1), generator=g).cuda()
    with torch.no_grad():
        assert model._step(ids, caches, 0) is not None
    x = model.tok_emb.weight[ids[:, 0]].double()
    want = (x - x.mean(-1, keepdim=True)) / torch.sqrt(x.var(-1, unbiased=False, keepdim=True) + 1e-5)
    got = caches[0][0][:, 0].reshape(B, C).double()
    assert ((got - want).abs() <= (2 * 2.0 ** -9 + C * 2.0 ** -24) * 1.01 * want.abs()).all()


@pytest.mark.parametrize("kind", ["rows", "row stride"])
def test_caches_past_the_limits_go_layer_by_layer(fa_lib, kind):
    """More rows, or rows further apart, than the one-launch step takes (0.5 and 4.3 GB a cache)."""
    model, _ = _model(64, 1, 1, 97, 64)
    shape, stride = ((1, (1 << 22) + 8, 1, 64), (64, 64, 64, 1)) if kind == "rows" else ((1, 2, 1, 64), (64, 1 << 31, 64, 1))
    far = [tuple(torch.empty_strided(shape, stride, dtype=torch.bfloat16, device="cuda") for _ in range(2))]
    near = model.allocate_kv_cache(1, 2)
    ids = torch.randint(0, 97, (1, 2), device="cuda")
    with torch.no_grad():
        model._step(ids[:, :1], near, 0)
        for a, b in zip(far[0], near[0]):
            a[:, 0] = b[:, 0]
        assert model._step(ids[:, 1:], far, 1) is None
        got = model(ids[:, 1:], kv_caches=far, pos=1).float()
        want = model(ids[:, 1:], kv_caches=near, pos=1).float()
    assert ((got - want).norm() / want.norm()).item() <= 2 * 2.0 ** -8 * math.sqrt(8 + 4)
