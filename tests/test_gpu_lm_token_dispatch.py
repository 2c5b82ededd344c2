"""What LadderLM hands to the generation kernel (csrc/lm_token.cu): models that ask for anything the
kernel does not compute go layer by layer, with the results and side effects that path has."""
import copy
import io

import pytest
import torch
import torch.nn as nn

from _gpu_cases import TOL, option
from elman_b200 import _lib
from elman_b200.ladder_lm import LadderLM
from oracle import elman_oracle as orc

pytestmark = pytest.mark.gpu

TOKENS = [[3], [250], [77]]


def _model(d=64, depth=2, seed=5, **kw):
    torch.manual_seed(seed)
    return LadderLM(vocab_size=256, dim=d, depth=depth, level=1, **{"r_h_mode": "none", **kw}).cuda().bfloat16().eval()


def _tokens():
    return torch.tensor(TOKENS).cuda()


@torch.no_grad()
def _one_token(model, tokens=None):
    """(logits, launches of the library)"""
    before = _lib.launch_count()
    logits = model(_tokens() if tokens is None else tokens)
    torch.cuda.synchronize()
    return logits, _lib.launch_count() - before


def _layer_by_layer(model, tokens=None):
    with option("rec_reg", 1):     # no register kernels: the generation kernel steps aside
        return _one_token(model, tokens)[0]


def _close(a, b):
    return a.shape == b.shape and orc.rel_err(a.float().cpu(), b.float().cpu()) < TOL[torch.bfloat16]


def test_plain_model_takes_the_kernel():
    model = _model()
    logits, launches = _one_token(model)
    assert launches <= 2 and _close(logits, _layer_by_layer(model))


@pytest.mark.parametrize("where", ["embedding", "norm", "W_h", "in_proj"])
def test_parametrised_weights_go_layer_by_layer(where):
    from torch.nn.utils import parametrizations, prune
    model = _model()
    if where == "W_h":
        prune.random_unstructured(model.layers[1].cell, "W_h", amount=0.5)
    elif where == "norm":
        prune.random_unstructured(model.norm, "weight", amount=0.5)
    else:
        parametrizations.weight_norm(model.embedding if where == "embedding" else model.layers[0].in_proj)
    logits, launches = _one_token(model)
    assert launches > 2 and _close(logits, _layer_by_layer(model))


def test_dropout_that_is_training_drops():
    model = _model(dropout=0.5)
    model.eval()
    assert torch.equal(_one_token(model)[0], _one_token(model)[0])
    for layer in model.layers:
        layer.dropout.train()          # Monte Carlo dropout
    assert not torch.equal(_one_token(model)[0], _one_token(model)[0])


def test_replaced_modules_are_called():
    class Halve(nn.Module):
        def forward(self, x):
            return 0.5 * x

    model = _model()
    plain, _ = _one_token(model)
    model.layers[0].dropout = Halve()
    logits, _ = _one_token(model)
    assert not torch.equal(logits, plain) and _close(logits, _layer_by_layer(model))


@pytest.mark.parametrize("kind", ["forward", "pre", "global"])
@pytest.mark.parametrize("where", ["embedding", "layers.1", "layers.0.cell", "layers.1.dropout"])
def test_hooks_fire(where, kind):
    model = _model(dropout=0.1)
    module, calls = model.get_submodule(where), []
    if kind == "forward":
        handle = module.register_forward_hook(lambda m, *a: calls.append(m))
    elif kind == "pre":
        handle = module.register_forward_pre_hook(lambda m, *a: calls.append(m))
    else:
        handle = nn.modules.module.register_module_forward_hook(
            lambda m, *a: calls.append(m) if m is module else None)
    try:
        _one_token(model)
    finally:
        handle.remove()
    assert calls == [module]


def test_residual_stream_in_the_models_own_type_is_kept():
    model = _model(d=256, depth=4)
    model.residual_in_fp32 = False
    _, launches = _one_token(model)
    assert launches > 2


def test_transposed_weight_is_read_as_the_tensor_says():
    model = _model()
    _one_token(model)
    W = model.layers[0].cell.W_x
    W.data = W.data.t()               # the same address
    logits, _ = _one_token(model)
    assert _close(logits, _layer_by_layer(model))
    model.layers[0].cell.W_x = nn.Parameter(W.detach().contiguous())
    assert _close(logits, _one_token(model)[0])


@pytest.mark.parametrize("rows", [264, 100])
def test_vocabulary_is_that_of_the_tables(rows):
    """Tables grown after construction (ids up to 263 are legal then), or cut."""
    model = _model()
    torch.manual_seed(1)
    model.embedding = nn.Embedding(rows, 64, device="cuda", dtype=torch.bfloat16)
    model.lm_head = nn.Linear(64, rows, bias=False, device="cuda", dtype=torch.bfloat16)
    tokens = torch.tensor([[3], [rows - 1]]).cuda()
    logits, _ = _one_token(model, tokens)
    assert logits.shape == (2, 1, rows)
    assert _lib.device_status()[0] == 0
    assert _close(logits, _layer_by_layer(model, tokens))
    assert _one_token(model, tokens)[1] <= 2


def test_tables_of_different_sizes_go_layer_by_layer():
    model = _model()
    model.lm_head = nn.Linear(64, 8, bias=False, device="cuda", dtype=torch.bfloat16)
    logits, launches = _one_token(model)
    assert launches > 2 and logits.shape == (3, 1, 8)


def test_model_is_copied_and_saved_after_a_token():
    model = _model()
    want, _ = _one_token(model)
    assert torch.equal(_one_token(copy.deepcopy(model))[0], want)
    buffer = io.BytesIO()
    torch.save(model, buffer)
    buffer.seek(0)
    assert torch.equal(_one_token(torch.load(buffer, weights_only=False))[0], want)


def test_forward_mode_is_refused_and_not_dropped():
    """The layers' autograd function has no forward derivative and says so."""
    model = _model()
    states = [torch.zeros(3, 64, dtype=torch.bfloat16, device="cuda") for _ in range(2)]
    with torch.no_grad(), torch.autograd.forward_ad.dual_level():
        states[0] = torch.autograd.forward_ad.make_dual(states[0], torch.ones_like(states[0]))
        with pytest.raises(RuntimeError):
            model(_tokens(), prev_hiddens=states)


def test_layers_that_share_a_cell_advance_its_vector_in_turn():
    model = _model(r_h_mode="spectral_norm", r_h_init_gain=1.0)
    model.layers[1] = model.layers[0]
    u = nn.functional.normalize(torch.randn(64, device="cuda"), dim=0).bfloat16()
    after = []
    for run in (_layer_by_layer, lambda m: _one_token(m)[0]):
        model.layers[0].cell._spectral_u = u.clone()
        run(model)
        after.append(model.layers[0].cell._spectral_u.float().cpu())
    assert torch.equal(after[0], after[1])


def test_vector_that_was_reset_is_drawn_again():
    model = _model(r_h_mode="spectral_norm", r_h_init_gain=1.0)
    _one_token(model)
    states = [torch.full((3, 64), 0.5, dtype=torch.bfloat16, device="cuda") for _ in range(2)]
    with torch.no_grad():
        want = model(_tokens(), prev_hiddens=states)
        for layer in model.layers:
            layer.cell._spectral_u = None
        got = model(_tokens(), prev_hiddens=states)
    assert all(layer.cell._spectral_u is not None for layer in model.layers)
    assert orc.rel_err(got.float().cpu(), want.float().cpu()) < 0.1    # another start of three iterations
