"""LadderLM's generation step in one kernel (csrc/lm_token.cu) against the same model layer by layer, at
the edges of its tiles: sequences around the 8-row tiles and the 32-row turns, widths that leave a CTA
or a warp's K range partly filled, with and without carried states, with and without spectral
normalisation.  Tolerance: the parity tests' bf16 2e-2 — both sides round activations to 8 bits six
times per layer."""
import ctypes
import threading

import pytest
import torch

from _gpu_cases import TOL, option
from elman_b200 import _lib
from elman_b200.ladder_lm import LadderLM
from oracle import elman_oracle as orc

pytestmark = pytest.mark.gpu


def _model(d, depth, mode):
    torch.manual_seed(d)
    return LadderLM(vocab_size=256, dim=d, depth=depth, level=1, r_h_mode=mode).cuda().bfloat16().eval()


@pytest.mark.parametrize("B,d,depth,mode", [(1, 1280, 3, "spectral_norm"), (8, 40, 2, "none"), (9, 264, 2, "none"),
                                            (17, 496, 3, "spectral_norm"), (33, 264, 2, "spectral_norm"),
                                            (64, 1024, 2, "none"), (3, 1368, 2, "spectral_norm")])
@pytest.mark.parametrize("carried", [True, False])
def test_one_token_matches_layer_by_layer(B, d, depth, mode, carried):
    model = _model(d, depth, mode)
    g = torch.Generator().manual_seed(B)
    tokens = torch.randint(0, 256, (B, 1), generator=g).cuda()
    states = [torch.tanh(torch.randn(B, d, generator=g)).bfloat16().cuda() for _ in range(depth)] if carried else None
    us = [torch.nn.functional.normalize(torch.randn(d, generator=g), dim=0).bfloat16().cuda() for _ in range(depth)]
    outs = []
    for off in (1, 0):
        for layer, u in zip(model.layers, us):
            layer.cell._spectral_u = u.clone()
        with torch.no_grad(), option("rec_reg", off):
            before = _lib.launch_count()
            logits, (hs, extra) = model(tokens, return_prev_hiddens=True, prev_hiddens=states)
            launches = _lib.launch_count() - before
        torch.cuda.synchronize()
        assert extra is None and logits.shape == (B, 1, 256) and all(h.shape == (B, d) for h in hs)
        outs.append([logits] + list(hs) + ([l.cell._spectral_u for l in model.layers] if mode != "none" else []))
    assert launches <= 3, "the generation kernel was not used"
    assert _lib.device_status()[0] == 0
    for a, b in zip(outs[1], outs[0]):
        assert orc.rel_err(a.float().cpu(), b.float().cpu()) < TOL[torch.bfloat16]


def test_changed_parameters_are_seen_and_a_token_outside_the_vocabulary_is_reported():
    model = _model(64, 2, "none")
    tok = torch.tensor([[3]]).cuda()
    with torch.no_grad():
        a = model(tok)
        model.layers[0].cell.W_x.mul_(0.5)                              # in place
        b = model(tok)
        model.layers[1].cell.W_x.data = model.layers[1].cell.W_x * 0.5   # another tensor
        c = model(tok)
        assert not torch.equal(a, b) and not torch.equal(b, c)
        model(torch.tensor([[256]]).cuda())
        torch.cuda.synchronize()
    code, detail = _lib.device_status(clear=True)
    assert code == 3 and detail >> 24 == 8


@pytest.mark.parametrize("mode,stall", [("none", 1), ("spectral_norm", 1), ("spectral_norm", 1000),
                                        ("spectral_norm", 1002)])
def test_gives_up_when_a_block_stalls_and_recovers(mode, stall):
    """A layer's input, and a round of the power iterations in front of it (1000 + its number)."""
    model = _model(64, 3, mode)
    tok = torch.tensor([[3], [5]]).cuda()
    us = [torch.full((64,), 0.125, dtype=torch.bfloat16, device="cuda") for _ in range(3)]

    def step():
        for layer, u in zip(model.layers, us):
            layer.cell._spectral_u = u.clone()
        return model(tok)

    with torch.no_grad():
        want = step()
        with option("spin_limit", 5000), option("test_stall_step", stall):
            step()
        torch.cuda.synchronize()
        code, detail = _lib.device_status(clear=True)
        assert code == 3 and detail >> 24 == 8
        assert torch.equal(step(), want)


def test_bias_between_two_words_goes_layer_by_layer():
    """Parameters packed into one flat buffer may start at any element; the kernel reads the bias in
    pairs of features.  A state buffer of a C caller that starts there is refused."""
    model = _model(64, 2, "none")
    tok = torch.tensor([[3], [5]]).cuda()
    with torch.no_grad():
        model.layers[0].cell.b.normal_()
        want = model(tok)
        flat = torch.empty(65, dtype=torch.bfloat16, device="cuda")
        flat[1:] = model.layers[0].cell.b
        model.layers[0].cell.b.data = flat[1:]
        before = _lib.launch_count()
        got = model(tok)
        assert _lib.launch_count() - before > 2
    assert orc.rel_err(got.float().cpu(), want.float().cpu()) < TOL[torch.bfloat16]
    lib, x = _lib.load(), torch.zeros(4096, dtype=torch.bfloat16, device="cuda")
    ws = torch.empty(lib.elman_e1_lm_token_workspace(1, 1, 32), dtype=torch.uint8, device="cuda")
    at = x.data_ptr()
    for bias, h_out in ((at + 2, at), (at, at + 2)):
        refs = (ctypes.c_void_p * 9)(at, at, at, at, bias, at, None, None, h_out)
        before = _lib.launch_count()
        rc = lib.elman_e1_lm_token(_lib.ELMAN_BF16, 1, 1, 32, 16, at, at, refs, at, at, 1e-6, 0.99, 1e-8,
                                   at, ws.data_ptr(), ws.numel(), torch.cuda.current_stream().cuda_stream)
        assert rc == _lib.ELMAN_ERR_UNSUPPORTED and _lib.launch_count() == before


def test_two_threads_at_two_widths():
    """Widths that share the kernels and differ in the shared memory they need: neither thread's launch
    depends on what the other one last asked for."""
    models = [_model(d, 2, "spectral_norm") for d in (1032, 1272)]
    tok = torch.tensor([[3]]).cuda()
    with torch.no_grad():
        for m in models:
            m(tok)
    torch.cuda.synchronize()
    errors = []

    def generate(model):
        try:
            with torch.no_grad(), torch.cuda.stream(torch.cuda.Stream()):
                for _ in range(400):
                    model(tok)
                torch.cuda.current_stream().synchronize()
        except Exception as e:
            errors.append(e)

    threads = [threading.Thread(target=generate, args=(m,)) for m in models]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors and _lib.device_status()[0] == 0
