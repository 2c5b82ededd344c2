"""Which models LadderLM hands to the generation kernel, on the CPU: what it reads out of the modules
(`_token_operands`), and that everything else reaches the layers."""
import pytest
import torch

from elman_b200.ladder_lm import LadderLM


def _model(level=1, **kw):
    return LadderLM(vocab_size=256, dim=32, depth=2, level=level, **kw).bfloat16().eval()


def _parametrise(model, where):
    from torch.nn.utils import parametrizations, prune
    if where == "W_h":
        prune.random_unstructured(model.layers[1].cell, "W_h", amount=0.5)
    elif where == "norm":
        prune.random_unstructured(model.norm, "weight", amount=0.5)
    else:
        parametrizations.weight_norm(model.get_submodule(where))


def test_plain_model():
    model = _model()
    params, eps, cells = model._token_operands()
    assert eps == torch.finfo(torch.float32).eps
    assert [p.shape for p in params] == (
        [(256, 32)] + 2 * [(32,), (64, 32), (32, 32), (32, 32), (32,), (32, 32)] + [(32,), (256, 32)])
    assert cells == [layer.cell for layer in model.layers]


@pytest.mark.parametrize("where", ["embedding", "norm", "W_h", "layers.0.in_proj", "lm_head"])
def test_parametrised_weights(where):
    model = _model()
    _parametrise(model, where)
    assert model._token_operands() is None


@pytest.mark.parametrize("level", [0, 1])
def test_one_token_on_the_cpu_is_refused_by_the_layer(level):
    model = _model(level)
    _parametrise(model, "embedding")
    with torch.no_grad(), pytest.raises(RuntimeError, match="CUDA"):
        model(torch.tensor([[3]]))


def test_dropout_that_is_training():
    model = _model(dropout=0.5)
    assert model._token_operands() is not None
    model.layers[1].dropout.train()             # the model itself still in eval()
    assert model._token_operands() is None
    model.train().layers[1].dropout.eval()
    assert model._token_operands() is None       # layer 0
    model.layers[0].dropout.eval()
    assert model._token_operands() is not None


def test_replaced_dropout():
    model = _model()
    model.layers[0].dropout = torch.nn.Tanh()
    assert model._token_operands() is None


@pytest.mark.parametrize("kind", ["forward", "pre", "global", "global pre"])
@pytest.mark.parametrize("where", ["embedding", "layers.1", "layers.0.cell", "layers.1.dropout"])
def test_hooks(where, kind):
    model = _model(dropout=0.1)
    module, hooks = model.get_submodule(where), torch.nn.modules.module
    register = {"forward": module.register_forward_hook, "pre": module.register_forward_pre_hook,
                "global": hooks.register_module_forward_hook,
                "global pre": hooks.register_module_forward_pre_hook}[kind]
    handle = register(lambda *a: None)
    try:
        assert model._token_operands() is None
    finally:
        handle.remove()
    assert model._token_operands() is not None


@pytest.mark.parametrize("where", ["embedding", "layers.1", "layers.0.cell", "layers.1.dropout"])
def test_other_classes_and_forwards_of_their_own(where):
    model = _model()
    module = model.get_submodule(where)
    module.forward = module.forward
    assert model._token_operands() is None
    del module.forward
    assert model._token_operands() is not None
    module.__class__ = type("Mine", (type(module),), {})
    assert model._token_operands() is None


def test_subclass_and_renormalised_embedding():
    model = _model()
    model.embedding.max_norm = 1.0
    assert model._token_operands() is None
    model = _model()
    model.__class__ = type("Mine", (LadderLM,), {})     # may override _add_norm, _head
    assert model._token_operands() is None


def test_tensors_in_another_form():
    model = _model()
    W = model.layers[0].cell.W_x
    W.data = W.data.t()                                   # same storage, same address
    assert model._token_operands() is None
    W.data = W.data.contiguous()
    assert model._token_operands() is not None
    model.layers[1].cell.b.data = model.layers[1].cell.b.data.float()
    assert model._token_operands() is None
    model = _model()
    model.layer_norms[1].eps = 1e-3
    assert model._token_operands() is None


def test_tables_of_another_size():
    nn, model = torch.nn, _model()
    model.lm_head = nn.Linear(32, 8, bias=False, dtype=torch.bfloat16)
    assert model._token_operands() is None
    model.embedding = nn.Embedding(8, 32, dtype=torch.bfloat16)
    assert model._token_operands()[0][0].shape == (8, 32)      # vocab_size is not asked
    model.embedding = nn.Embedding(8, 40, dtype=torch.bfloat16)
    assert model._token_operands() is None


@pytest.mark.parametrize("name,shape", [("layers.0.cell.W_x", (32, 40)), ("layers.1.cell.b", (64,)),
                                        ("layers.0.in_proj.weight", (32, 32)), ("layer_norms.1.weight", (8,)),
                                        ("norm.weight", (1, 32)), ("layers.1.out_proj.weight", (32, 16))])
def test_weights_of_another_shape(name, shape):
    model = _model()
    model.get_parameter(name).data = torch.zeros(shape, dtype=torch.bfloat16)
    assert model._token_operands() is None


def test_fewer_layers_than_it_was_built_with():
    model = _model()
    model.layers = model.layers[:1]
    assert model._token_operands() is None                      # two norms, one layer
    model.layer_norms = model.layer_norms[:1]
    assert len(model._token_operands()[2]) == 1
    assert _model(expansion=1.5)._token_operands() is None


def test_residual_stream_in_the_models_own_type():
    model = _model()
    model.residual_in_fp32 = False
    assert model._token_operands() is None


def test_transforms_of_the_call():
    model, seen = _model(), []

    def look(x):
        seen.append(model._token_operands())
        return x

    torch.func.vmap(look)(torch.zeros(2))
    with torch.autograd.forward_ad.dual_level():
        look(None)
    torch.jit.trace(look, torch.zeros(2), check_trace=False)
    assert seen == [None, None, None]
    assert model._token_operands() is not None
