"""The workloads this package is measured on.

A case is a dict of plain values: `path` names the entry point, the rest are its sizes.  The paths
are the ways a program uses the package:

  generate   one more token for every running sequence through `LadderLM` (states carried)
  prompt     a whole prompt through `LadderLM` without gradients, states kept for generation
  step       one optimizer step of `LadderLM` through `GraphedTrainStep`
  layer      `MambaGatedElman` forward and backward under autograd
  e1 e0 e5   a cell forward and backward through the extension-module functions
  e1_forward the E1 cell without a backward pass

`listed()` are the fixed cases, `draw()` gives more of the same ranges.
"""
import math

import torch

from elman_b200 import hasty_pytorch_lib as H
from elman_b200.ladder_lm import LadderLM
from elman_b200.mamba_gated_elman import MambaGatedElman
from elman_b200.train_step import FlatAdamW, GraphedTrainStep, make_gradient_reducer

VOCAB = 256
DTYPES = {"bf16": torch.bfloat16, "f32": torch.float32}


def listed():
    return [
        # interactive generation from the byte-level model: one sequence, one token per call
        dict(name="generate_one", path="generate", dtype="bf16", B=1, T=1, d=1280, depth=6),
        # generation for a set of users at once, of a number that nobody rounded
        dict(name="generate_batch", path="generate", dtype="bf16", B=27, T=1, d=1280, depth=6),
        # reading a few prompts before generation, of a length that is not a round number
        dict(name="prompt", path="prompt", dtype="bf16", B=3, T=333, d=1280, depth=6),
        # training the byte-level model: the whole optimizer step
        dict(name="train_step", path="step", dtype="bf16", B=32, T=512, d=1280, depth=6),
        # one E1 layer as a module of somebody's own model, inner width 1.5 times the outer one
        dict(name="layer", path="layer", dtype="bf16", B=48, T=256, d=512, expansion=1.5),
        # the E1 cell at the size the package is quoted on
        dict(name="e1_cell", path="e1", dtype="bf16", B=32, T=512, d=1280),
        # the E1 cell at a width and a batch that come from a parameter budget and from what is
        # left of a data set, not from the hardware
        dict(name="e1_ragged", path="e1", dtype="bf16", B=37, T=200, d=952),
        # the single-precision cell at the small configuration that parity is checked on
        dict(name="e1_f32", path="e1", dtype="f32", B=4, T=128, d=256),
        # E0 in a mid-sized model
        dict(name="e0_cell", path="e0", dtype="bf16", B=48, T=256, d=768),
        # E5 at its quoted size, and at a batch nearer to the one its models were trained with
        dict(name="e5_cell", path="e5", dtype="bf16", B=32, T=512, d=1536, r=270),
        dict(name="e5_batch", path="e5", dtype="bf16", B=128, T=160, d=1536, r=270),
        # scoring long sequences in bulk: wide layer, large batch, forward only
        dict(name="e1_wide_forward", path="e1_forward", dtype="bf16", B=256, T=2048, d=2048),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _width(rng, lo, hi):
    """Mostly the multiples of 64 that configurations use, sometimes any multiple of 8."""
    step = rng.choice([128, 64, 64, 8])
    return max(lo, int(round(_log_int(rng, lo, hi) / step)) * step)


def _length(rng, lo, hi, B, d):
    """A sequence length whose recurrence is no more work than that of the large listed cases."""
    return min(_log_int(rng, lo, hi), max(8, int(2.2e10 / (B * d * d))))


def draw(rng):
    path = rng.choice(["generate", "prompt", "step", "layer", "e1", "e1", "e0", "e5", "e1_forward"])
    if path == "generate":
        return dict(path=path, dtype="bf16", B=_log_int(rng, 1, 64), T=1, d=_width(rng, 256, 1280),
                    depth=rng.randint(2, 8))
    if path == "prompt":
        return dict(path=path, dtype="bf16", B=_log_int(rng, 1, 8), T=_log_int(rng, 16, 512),
                    d=_width(rng, 256, 1280), depth=rng.randint(2, 6))
    if path == "step":
        return dict(path=path, dtype="bf16", B=_log_int(rng, 4, 32), T=_log_int(rng, 64, 512),
                    d=128 * rng.randint(2, 10), depth=rng.randint(2, 6))
    if path == "layer":
        B, d, expansion = _log_int(rng, 1, 48), _width(rng, 256, 1024), rng.choice([1.0, 1.0, 1.5, 2.0])
        return dict(path=path, dtype="bf16", B=B, T=_length(rng, 16, 512, B, int(d * expansion)), d=d,
                    expansion=expansion)
    if path == "e1" and rng.random() < 0.4:
        return dict(path=path, dtype="f32", B=_log_int(rng, 1, 16), T=_log_int(rng, 16, 256),
                    d=_width(rng, 64, 512))
    if path in ("e1", "e0"):
        B, d = _log_int(rng, 1, 64), _width(rng, 256, 1536)
        return dict(path=path, dtype="bf16", B=B, T=_length(rng, 16, 512, B, d), d=d)
    if path == "e5":
        d = _width(rng, 512, 1536)
        return dict(path=path, dtype="bf16", B=_log_int(rng, 4, 128), T=_log_int(rng, 16, 128), d=d,
                    r=rng.randint(d // 8, d // 6))
    return dict(path=path, dtype="bf16", B=_log_int(rng, 32, 256), T=_log_int(rng, 64, 1024),
                d=128 * rng.randint(4, 16))


# ------------------------------------------------------------------------------- inputs

class _Inputs:
    """Seeded tensors on the GPU: activations N(0,1), weights scaled by their fan-in, the
    recurrent matrix with spectral radius 0.9."""

    def __init__(self, case, seed):
        self.dtype = DTYPES[case["dtype"]]
        self.rng = torch.Generator(device="cuda").manual_seed(seed)

    def normal(self, *shape, scale=1.0):
        t = torch.randn(*shape, generator=self.rng, device="cuda", dtype=self.dtype)
        return t if scale == 1.0 else t.mul_(scale)

    def dense(self, d):
        return self.normal(d, d, scale=1 / math.sqrt(d))

    def recurrent(self, d):
        return self.normal(d, d, scale=0.9 / math.sqrt(d))   # circular law: radius 0.9

    def bytes(self, B, T):
        """Byte values with the skewed frequencies of text (Zipf, s = 1.1)."""
        p = torch.arange(1, VOCAB + 1, dtype=torch.float32, device="cuda") ** -1.1
        return torch.multinomial(p, B * T, replacement=True, generator=self.rng).view(B, T)


def _model(case, seed, **kw):
    torch.manual_seed(seed)
    with torch.device("cuda"):
        model = LadderLM(vocab_size=VOCAB, dim=case["d"], depth=case["depth"], level=1, **kw)
    return model.to(DTYPES[case["dtype"]])


def prepare(case, seed):
    new = _Inputs(case, seed)
    path, B, T, d = case["path"], case["B"], case["T"], case["d"]
    s = {"path": path}
    if path in ("generate", "prompt"):
        s["model"] = _model(case, seed).eval()
        s["tokens"] = new.bytes(B, T)
        # generation carries the states of what was read before
        s["hiddens"] = ([new.normal(B, d).tanh_() for _ in range(case["depth"])]
                        if path == "generate" else None)
    elif path == "step":
        model = _model(case, seed, pipeline_chunks=10)
        grads = make_gradient_reducer(model)
        # the learning rate of a schedule's warm-up
        opt = FlatAdamW(grads, lr=1e-5, betas=(0.9, 0.95), eps=1e-8, weight_decay=0.1)
        s["tokens"] = new.bytes(B, T + 1)
        s["step"] = GraphedTrainStep(model, opt, s["tokens"], max_grad_norm=1.0,
                                     autocast_dtype=torch.bfloat16, reducer=grads)
        s["opt"], s["model"] = opt, model
    elif path == "layer":
        torch.manual_seed(seed)
        with torch.device("cuda"):
            layer = MambaGatedElman(d, expansion=case["expansion"], r_h_init_gain=0.5)
        s["layer"] = layer.to(new.dtype).train()
        s["x"] = new.normal(B, T, d).requires_grad_()
        s["dy"] = new.normal(B, T, d)
    else:
        s["x"], s["h0"], s["b"] = new.normal(T, B, d), new.normal(B, d).tanh_(), new.normal(d, scale=0.1)
        if path == "e5":
            r = case["r"]
            k = 1 / math.sqrt(math.sqrt(d * r))      # U V of unit gain where rank allows
            s["factors"] = [new.normal(*((d, r) if i % 2 == 0 else (r, d)),
                                       scale=k * (0.9 if i < 2 else 1.0)) for i in range(6)]
        else:
            s["W_x"], s["W_h"] = new.dense(d), new.recurrent(d)
        if path == "e0":
            s["W_gate"], s["b_gate"] = new.dense(d), new.normal(d, scale=0.1)
        elif path != "e5":
            s["z"] = new.normal(T, B, d)
        if path != "e1_forward":
            s["dy"] = new.normal(T, B, d)
    return s


# --------------------------------------------------------------------------------- a pass

def run(s):
    return _RUN[s["path"]](s)


def _run_lm(s):
    with torch.no_grad():
        logits, (hiddens, _) = s["model"](s["tokens"], return_prev_hiddens=True,
                                          prev_hiddens=s["hiddens"])
    return {"logits": logits, "hiddens": hiddens}


def _run_step(s):
    loss = s["step"](s["tokens"])
    return {"loss": loss, "params": s["opt"].flat_params,
            "grads": [p.grad for p in s["model"].parameters()]}


def _run_layer(s):
    layer, x = s["layer"], s["x"]
    params = list(layer.parameters())
    out, h_final = layer(x)
    grads = torch.autograd.grad(out, [x] + params, s["dy"])
    return {"out": out.detach(), "h_final": h_final.detach(), "grads": grads}


def _run_e1(s):
    h, out, v = H.mamba_gated_elman_forward(True, s["x"], s["z"], s["h0"], s["W_x"], s["W_h"], s["b"])
    return [h, out, v] + H.mamba_gated_elman_backward(s["W_x"], s["W_h"], s["x"], s["z"], h, v, s["dy"])


def _run_e1_forward(s):
    h, out, _ = H.mamba_gated_elman_forward(False, s["x"], s["z"], s["h0"], s["W_x"], s["W_h"], s["b"])
    return [h, out]


def _run_e0(s):
    h, out, v, gate = H.stock_elman_forward(True, s["x"], s["h0"], s["W_x"], s["W_h"], s["W_gate"],
                                            s["b"], s["b_gate"])
    return [h, out, v, gate] + H.stock_elman_backward(s["W_x"], s["W_h"], s["W_gate"], s["x"], h, v,
                                                      gate, s["dy"])


def _run_e5(s):
    f = s["factors"]
    h, out, v = H.pure_lowrank_elman_forward(True, s["x"], s["h0"], *f, s["b"])
    return [h, out, v] + H.pure_lowrank_elman_backward(*f, s["x"], h, v, s["dy"])


_RUN = {"generate": _run_lm, "prompt": _run_lm, "step": _run_step, "layer": _run_layer,
        "e1": _run_e1, "e1_forward": _run_e1_forward, "e0": _run_e0, "e5": _run_e5}


# ------------------------------------------------------------------------ work, tolerance

def work(case):
    """Bytes and operations of one pass that no implementation can do without: every input and
    weight read once, every output and gradient written once; matrix products at 2 per
    multiply-add."""
    path, B, T, d = case["path"], case["B"], case["T"], case["d"]
    e = 4 if case["dtype"] == "f32" else 2
    n = T * B * d                                   # elements of one [T,B,d] tensor
    if path in ("generate", "prompt", "step"):
        L, tb = case["depth"], T * B
        weights = L * (5 * d * d + 2 * d) + VOCAB * d + d
        flops = 2 * tb * (L * 5 * d * d + VOCAB * d)
        if path == "step":
            # forward and both backward products; parameters and the two moments read and
            # written, gradients written
            return {"bytes": 7 * weights * e + tb * 8, "flops": 3 * flops}
        return {"bytes": (weights + tb * VOCAB + L * (2 if path == "generate" else 1) * B * d) * e + tb * 8,
                "flops": flops}
    if path == "layer":
        di = int(d * case["expansion"])
        weights = 3 * d * di + 2 * di * di
        return {"bytes": (4 * T * B * d + 2 * weights) * e, "flops": 6 * T * B * weights}
    if path == "e5":
        r = case["r"]
        # x and dy in, h, out, v and dx out; three factor pairs in, their gradients out
        return {"bytes": (6 * n + 2 * 6 * d * r) * e, "flops": 3 * 2 * T * B * 6 * d * r}
    if path == "e0":
        return {"bytes": (7 * n + 2 * 3 * d * d) * e, "flops": 3 * 2 * T * B * 3 * d * d}
    if path == "e1":
        # x, z and dy in; h, out, v, dx and dz out
        return {"bytes": (8 * n + 2 * 2 * d * d) * e, "flops": 3 * 2 * T * B * 2 * d * d}
    return {"bytes": (4 * n + 2 * d * d) * e, "flops": 2 * T * B * 2 * d * d}


def tolerance(case):
    """bf16: states and gradients are rounded to 8 bits at every step of a recurrence that feeds
    them back, in a model once more per layer; fp32: sums of a thousand terms, fed back as well."""
    if case["dtype"] == "f32":
        return {"rel": 1e-5}
    return {"rel": 2e-2 if "depth" in case else 1e-2}
