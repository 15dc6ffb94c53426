"""What the paths past a model's modules are made from (step.ModelWatch, step.plain_modules), without a
GPU: every replacement that the modules' own forward would follow is seen, nothing else is."""
import copy

import pytest
import torch
import torch.nn as nn
import torch.nn.utils.prune

from tfg_flashattention_b200 import gpt2
from tfg_flashattention_b200.step import ModelWatch, StepPlan, plain_modules


def _model():
    cfg = {"vocab_size": 97, "context_length": 16, "emb_dim": 64, "n_heads": 1, "n_layers": 3, "drop_rate": 0.0,
           "qkv_bias": True, "impl_type": "cuda"}
    return gpt2.GPTModel(cfg, dtype=torch.bfloat16).eval().prepare_for_inference()


def _adapter(linear):
    class Adapter(nn.Linear):
        pass
    new = Adapter(linear.in_features, linear.out_features, bias=linear.bias is not None, dtype=torch.bfloat16)
    new.load_state_dict(linear.state_dict())
    return new


REPLACED = {
    "parameter": lambda m: setattr(m.trf_blocks[1].ff.layers[0], "bias", nn.Parameter(torch.zeros(256, dtype=torch.bfloat16))),
    "storage": lambda m: setattr(m.trf_blocks[1].norm2.scale, "data", torch.ones(64, dtype=torch.bfloat16)),
    "out_proj": lambda m: setattr(m.trf_blocks[2].att, "out_proj", nn.Linear(64, 64, dtype=torch.bfloat16)),
    "second mlp layer": lambda m: m.trf_blocks[0].ff.layers.__setitem__(2, nn.Linear(256, 64, dtype=torch.bfloat16)),
    "norm": lambda m: setattr(m.trf_blocks[0], "norm1", gpt2.LayerNorm(m.cfg)),
    "final norm": lambda m: setattr(m, "final_norm", gpt2.LayerNorm(m.cfg)),
    "head": lambda m: setattr(m, "out_head", nn.Linear(64, 97, bias=False, dtype=torch.bfloat16)),
    "embedding": lambda m: setattr(m, "tok_emb", nn.Embedding(97, 64, dtype=torch.bfloat16)),
    "block": lambda m: m.trf_blocks.__setitem__(1, copy.deepcopy(m.trf_blocks[1])),
    "fewer blocks": lambda m: m.trf_blocks.__delitem__(2),
    "more blocks": lambda m: m.trf_blocks.append(copy.deepcopy(m.trf_blocks[0])),
    "other order": lambda m: setattr(m, "trf_blocks", nn.Sequential(*reversed(m.trf_blocks))),
    "fused again": lambda m: m.trf_blocks[1].att.fuse_qkv(),
    "eps": lambda m: setattr(m.trf_blocks[1].norm1, "eps", 1e-3),
    "implementation": lambda m: setattr(m.trf_blocks[1].att, "impl_type", "manual"),
    "pruned": lambda m: torch.nn.utils.prune.l1_unstructured(m.trf_blocks[1].ff.layers[0], "weight", 0.5),
}


@pytest.mark.parametrize("what", REPLACED)
def test_replacements_are_seen(what):
    model = _model()
    watch = ModelWatch(model)
    assert watch.holds(model)
    REPLACED[what](model)
    assert not watch.holds(model)
    assert StepPlan.make(model) is None                  # (not on a GPU; and whatever was replaced, no error)


def test_what_is_no_replacement():
    model = _model()
    watch = ModelWatch(model)
    with torch.no_grad():
        model.trf_blocks[0].att.out_proj.weight.add_(1)  # values are read where they are
    model.to("cpu").requires_grad_(False)
    model.load_state_dict(model.state_dict())
    model.trf_blocks[0].att.W_query.bias = None          # (its part of the fused projection is what is used)
    assert watch.holds(model)


def test_modules_of_other_kinds():
    assert plain_modules(_model())
    for change in (lambda m: setattr(m.trf_blocks[0].att, "out_proj", _adapter(m.trf_blocks[0].att.out_proj)),
                   lambda m: m.trf_blocks[0].ff.layers.__setitem__(2, _adapter(m.trf_blocks[0].ff.layers[2])),
                   lambda m: setattr(m.trf_blocks[1].att, "impl_type", "manual"),
                   lambda m: setattr(m.trf_blocks[1].norm1, "eps", 1e-3),
                   lambda m: setattr(m.trf_blocks[1].att, "num_heads", 2),
                   lambda m: setattr(m, "out_head", _adapter(m.out_head)),
                   lambda m: torch.nn.utils.parametrizations.weight_norm(m.trf_blocks[0].ff.layers[0])):
        model = _model()
        change(model)
        assert not plain_modules(model)


@pytest.mark.parametrize("pick", [lambda m: m.tok_emb, lambda m: m.trf_blocks[0].att, lambda m: m.trf_blocks[2].ff,
                                  lambda m: m.trf_blocks[1].att.out_proj, lambda m: m.trf_blocks[1].ff.layers[2]])
def test_calls_that_somebody_waits_for(pick):
    model = _model()
    watch = ModelWatch(model)
    for register in (pick(model).register_forward_hook, pick(model).register_forward_pre_hook,
                     nn.modules.module.register_module_forward_hook):
        assert not watch.hooked()
        handle = register(lambda *a: None)
        assert watch.hooked() and watch.holds(model)
        handle.remove()
    pick(model).forward = lambda *a, **k: None           # of this module alone
    assert not watch.holds(model) and not plain_modules(model)


def test_copies_of_a_model_make_their_own():
    """A copy must not take over what belongs to the original's addresses, nor a watch over dictionaries that are
    no module's: whether it is pickled, copied, or a replica that shares all attributes but the modules."""
    import io
    model = _model()
    model._fused_blocks = True                           # (of a model on a GPU)
    seen = []
    make = lambda m: (seen.append(m), object())[1]
    mine = model._from_modules("x", make)
    assert model._from_modules("x", make) is mine and seen == [model]
    buffer = io.BytesIO()
    torch.save(model, buffer)
    buffer.seek(0)
    replica = model._replicate_for_data_parallel()
    replica._modules = dict(model._modules)
    for other in (copy.deepcopy(model), torch.load(buffer, weights_only=False), replica):
        assert other._from_modules("x", make) is not mine and seen[-1] is other
    with torch.no_grad():
        ids = torch.zeros(1, 4, dtype=torch.long)
        for m in (model, copy.deepcopy(model)):
            m._fused_blocks = False
            for blk in m.trf_blocks:
                blk.att.impl_type = "manual"
        assert copy.deepcopy(model)(ids).shape == (1, 4, 97)
