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
