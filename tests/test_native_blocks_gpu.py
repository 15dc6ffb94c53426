"""The binding's native loop over the blocks of a prompt against the same loop in Python: the same
operations and library algorithms in the same order, so the results are equal to the bit."""
import pytest
import torch

from tfg_flashattention_b200 import gpt2

pytestmark = pytest.mark.gpu


def _model(width=256, layers=3, bias=True):
    cfg = {"vocab_size": 503, "context_length": 400, "emb_dim": width, "n_heads": width // 64, "n_layers": layers,
           "drop_rate": 0.0, "qkv_bias": bias, "impl_type": "cuda"}
    return gpt2.init_random(gpt2.GPTModel(cfg, dtype=torch.bfloat16), seed=5, std=0.05).cuda().eval().prepare_for_inference()


@pytest.mark.parametrize("B,n,cached,last,bias", [(1, 2, True, True, True), (1, 129, False, False, False),
                                                  (3, 200, True, True, True), (2, 1, False, False, True)])
def test_native_loop_equals_python_loop(fa_lib, torch_binding, B, n, cached, last, bias):
    if torch_binding is None:
        pytest.skip("the torch extension binding could not be built here")
    model = _model(bias=bias)
    ids = torch.randint(0, 503, (B, n), device="cuda")
    caches = [model.allocate_kv_cache(B, n + 7) if cached else None for _ in range(2)]
    with torch.no_grad():
        x = torch.zeros(B, n, 256, dtype=torch.bfloat16, device="cuda")
        assert model._native_blocks(x, caches[0], 0) is not None
        got = model(ids, last_token_only=last, kv_caches=caches[0])
        model._native_blocks = lambda *a: None
        want = model(ids, last_token_only=last, kv_caches=caches[1])
    assert torch.equal(got, want)
    if cached:
        for a, b in zip(*caches):
            for t, r in zip(a, b):
                assert torch.equal(t, r) and t[:, :n].abs().sum() > 0 and (t[:, n:] == 0).all()


def test_native_loop_steps_aside(fa_lib, torch_binding):
    """Gradients, hooks, another position or other caches go through the modules as before; a replaced
    parameter is used."""
    if torch_binding is None:
        pytest.skip("the torch extension binding could not be built here")
    model = _model()
    ids = torch.randint(0, 503, (2, 40), device="cuda")
    x = torch.zeros(2, 40, 256, dtype=torch.bfloat16, device="cuda")
    assert model._native_blocks(x, None, 0) is None                          # gradients on
    with torch.no_grad():
        assert model._native_blocks(x, None, 0) is not None
        assert model._native_blocks(x, None, 1) is None
        assert model._native_blocks(x, model.allocate_kv_cache(2, 64, dtype=torch.float32), 0) is None
        seen = []
        handle = model.trf_blocks[1].ff.register_forward_hook(lambda *a: seen.append(1))
        before = model(ids)
        assert seen
        handle.remove()
        assert torch.equal(model(ids), before)
        model.trf_blocks[0].ff.layers[0].bias = torch.nn.Parameter(model.trf_blocks[0].ff.layers[0].bias + 1)
        changed = model(ids)
        model._native_blocks = lambda *a: None
        assert not torch.equal(changed, before) and torch.equal(model(ids), changed)


@pytest.mark.parametrize("change", ["out_proj", "second mlp layer", "adapter", "head", "final norm", "fewer blocks",
                                    "other order", "impl_type", "moved"])
def test_replaced_modules_are_used(fa_lib, torch_binding, change):
    """Prompts and single-token steps of a model whose modules were replaced after it was prepared, against a
    model of the same modules that is prepared then."""
    import copy
    import torch.nn as nn
    bf = dict(dtype=torch.bfloat16, device="cuda")

    class Adapter(nn.Linear):
        def forward(self, x):
            return super().forward(x) + 0.25 * x

    def apply(m):
        torch.manual_seed(11)
        blk = m.trf_blocks[1]
        if change == "out_proj":
            blk.att.out_proj = nn.Linear(256, 256, **bf)
        elif change == "second mlp layer":
            blk.ff.layers[2] = nn.Linear(1024, 256, **bf)
        elif change == "adapter":
            new = Adapter(256, 256, **bf)
            new.load_state_dict(blk.att.out_proj.state_dict())
            blk.att.out_proj = new
        elif change == "head":
            m.out_head = nn.Linear(256, 503, bias=False, **bf)
        elif change == "final norm":
            m.final_norm = gpt2.LayerNorm(m.cfg).cuda().bfloat16()
            with torch.no_grad():
                m.final_norm.shift.fill_(0.5)
        elif change == "fewer blocks":
            m.trf_blocks = m.trf_blocks[:2]
        elif change == "other order":
            m.trf_blocks = nn.Sequential(*reversed(m.trf_blocks))
        elif change == "impl_type":
            blk.att.impl_type = "manual"
        else:
            m.to("cuda")

    model, fresh = _model(), _model()
    caches = model.allocate_kv_cache(2, 32)
    ids = torch.randint(0, 503, (2, 20), device="cuda")
    with torch.no_grad():
        model(ids[:, :19], kv_caches=caches, pos=0)
        old = model(ids[:, 19:], kv_caches=caches, pos=19)
    apply(model)
    apply(fresh)
    fresh.prepare_for_inference()
    model._head_w = fresh._head_w                        # the padded copy for long prompts is prepare's own
    # as the modules themselves have it: no path past them
    fresh._native_blocks = lambda *a: None
    fresh._step = lambda *a, **k: None
    with torch.no_grad():
        got_caches, want_caches = model.allocate_kv_cache(2, 32), model.allocate_kv_cache(2, 32)
        got = model(ids[:, :19], kv_caches=got_caches, pos=0)
        want = fresh(ids[:, :19], kv_caches=want_caches, pos=0)
        assert torch.equal(got, want)
        got = model(ids[:, 19:], kv_caches=got_caches, pos=19).float()
        want = fresh(ids[:, 19:], kv_caches=want_caches, pos=19).float()
    # three layers of the one-launch step's and the modules' own roundings, see test_gpt_step_gpu.py
    assert ((got - want).norm() / want.norm()).item() <= 2 * 2.0 ** -8 * (8 * 3 + 4) ** 0.5
    if change == "moved":
        assert torch.equal(got, old.float()) and model._step_plan is not None and model._native_blocks(
            torch.zeros(2, 3, 256, **bf), None, 0) is None    # (gradients on)
    elif change != "impl_type":
        assert not torch.equal(got, old.float())


@pytest.mark.parametrize("kind", ["one prompt for four", "head first", "every third column", "row of 66", "misaligned"])
def test_caches_that_only_the_modules_write(fa_lib, torch_binding, kind):
    """Caches that the copy of the Python loop takes and the cache kernel does not: the loop steps aside and the
    result is the Python loop's."""
    if torch_binding is None:
        pytest.skip("the torch extension binding could not be built here")
    model = _model()
    B, n, H = (1 if kind == "one prompt for four" else 2), 20, 4
    ids = torch.randint(0, 503, (B, n), device="cuda")

    def cache():
        zeros = lambda *s: torch.zeros(*s, dtype=torch.bfloat16, device="cuda")
        if kind == "one prompt for four":
            return zeros(4, 32, H, 64)
        if kind == "head first":                         # (this one the kernel takes, too)
            return zeros(B, H, 32, 64).transpose(1, 2)
        if kind == "every third column":
            return zeros(B, 32, H, 192)[..., ::3]
        if kind == "row of 66":
            return zeros(B, 32, H, 66)[..., :64]
        return zeros(B * 32 * H * 64 + 4)[4:].view(B, 32, H, 64)

    caches = [[(cache(), cache()) for _ in range(3)] for _ in range(2)]
    x = torch.zeros(B, n, 256, dtype=torch.bfloat16, device="cuda")
    with torch.no_grad():
        assert (model._native_blocks(x, caches[0], 0) is not None) == (kind == "head first")
        got = model(ids, kv_caches=caches[0], pos=0)
        model._native_blocks = lambda *a: None
        want = model(ids, kv_caches=caches[1], pos=0)
    assert torch.equal(got, want)
    for a, b in zip(*caches):
        for t, r in zip(a, b):
            assert torch.equal(t, r) and (t[:, :n].abs().sum((1, 2, 3)) > 0).all()


@pytest.mark.parametrize("width,B,n", [(320, 1, 73), (320, 3, 5), (64, 1, 1), (448, 1, 129), (256, 1, 73)])
def test_native_loop_of_odd_heads_and_rows(fa_lib, torch_binding, width, B, n):
    """An odd number of heads times an odd number of rows: parts of one buffer that are 128-byte aligned only
    if nothing sees to it."""
    if torch_binding is None:
        pytest.skip("the torch extension binding could not be built here")
    model = _model(width=width, layers=2)
    ids = torch.randint(0, 503, (B, n), device="cuda")
    with torch.no_grad():
        assert model._native_blocks(torch.zeros(B, n, width, dtype=torch.bfloat16, device="cuda"), None, 0) is not None
        got = model(ids)
        model._native_blocks = lambda *a: None
        want = model(ids)
    assert torch.equal(got, want)


@pytest.mark.parametrize("offset", [8, 16, 64])
def test_native_loop_of_weights_in_a_flat_buffer(fa_lib, torch_binding, offset):
    """Parameters that are views into one buffer, 16, 32 and 128 bytes behind a 256-byte boundary.  The GEMMs'
    algorithms depend on it and sum in their own orders: a rounding to bf16 (2^-9) on either side for each
    of the eight per layer, taken as independent."""
    if torch_binding is None:
        pytest.skip("the torch extension binding could not be built here")
    model = _model(layers=2)
    for p in model.parameters():
        flat = torch.zeros(p.numel() + offset, dtype=torch.bfloat16, device="cuda")
        flat[offset:] = p.detach().flatten()
        p.data = flat[offset:].view(p.shape)
        assert p.data_ptr() % 256 == 2 * offset
    ids = torch.randint(0, 503, (2, 37), device="cuda")
    with torch.no_grad():
        assert model._native_blocks(torch.zeros(2, 37, 256, dtype=torch.bfloat16, device="cuda"), None, 0) is not None
        got = model(ids).float()
        model._native_blocks = lambda *a: None
        want = model(ids).float()
    assert ((got - want).norm() / want.norm()).item() <= 2 * 2.0 ** -9 * (8 * 2 + 4) ** 0.5


def test_no_blocks_and_another_device(fa_lib, torch_binding):
    """A model without blocks (all cut away) still gives its logits, with caches or without; input that is not
    where the weights are is left to the modules, which refuse it."""
    model = _model()
    ids = torch.randint(0, 503, (2, 9), device="cuda")
    with torch.no_grad():
        assert model._native_blocks(torch.zeros(2, 9, 256, dtype=torch.bfloat16), None, 0) is None
        model.trf_blocks = model.trf_blocks[:0]
        x = model.tok_emb(ids) + model.pos_emb(torch.arange(9, device="cuda"))
        want = torch.nn.functional.linear(model.final_norm(x), model.out_head.weight).float()
        for caches in (None, []):
            got = model(ids, kv_caches=caches).float()
            assert ((got - want).norm() / want.norm()).item() <= 2 * 2.0 ** -8
