"""The dense recurrence whose batch groups take turns on one set of CTAs (csrc/rec_turns.cuh), which
callers that overlap launches ask for with ELMAN_FLAG_COMPACT: batches that leave the last group or
the last set of groups partly filled (down to one row and one group), widths that leave a CTA, a
warp's K range or a block of 32 columns partly filled, every register split; against the CPU oracle
with the bf16 tolerance of the other parity tests."""
import pytest
import torch

from _gpu_cases import TOL, assert_close, errors, launches_of, option, oracle_e1, round_inputs
from elman_b200 import _lib
from elman_b200 import hasty_pytorch_lib as H
from oracle import elman_oracle as orc

pytestmark = pytest.mark.gpu


def run_compact(inp, flags=H.FLAG_COMPACT):
    dev, ref = round_inputs(inp, torch.bfloat16)
    h, out, v = H.mamba_gated_elman_forward(True, dev["x"], dev["z"], dev["h0"], dev["W_x"], dev["W_h"],
                                            dev["b"], flags)
    dx, dz, dWx, dWh, db, _ = H.mamba_gated_elman_backward_carry(
        dev["W_x"], dev["W_h"], dev["x"], dev["z"], h, v, dev["d_output"], None, flags)
    torch.cuda.synchronize()
    return dict(h=h, output=out, v=v, dx=dx, dz=dz, dW_x=dWx, dW_h=dWh, db=db), ref


@pytest.mark.parametrize("T,B,d", [(5, 9, 1280), (4, 33, 952), (5, 64, 520), (3, 61, 1000), (3, 17, 2040),
                                   (4, 20, 1536), (3, 24, 1800), (6, 48, 264), (5, 40, 768), (6, 20, 768),
                                   (1, 24, 1280)])
def test_ragged_shapes_match_oracle(T, B, d):
    inp = orc.make_e1_inputs(T, B, d, seed=5 * d + B)
    blocks = H.recurrence_blocks(torch.bfloat16, T, B, d, H.FLAG_COMPACT)
    assert 0 < blocks <= H.recurrence_blocks(torch.bfloat16, T, B, d)
    assert blocks < (B + 7) // 8 * ((d + 63) // 64), "several groups on one set of CTAs"
    with launches_of("rec_turns", 2):
        got, ref = run_compact(inp)
    assert _lib.device_status()[0] == 0
    assert_close(errors(got, oracle_e1(ref)), TOL[torch.bfloat16], f"T{T} B{B} d{d}")


@pytest.mark.parametrize("T,B,d,kernel", [(4, 65, 64, "rec_reg"), (3, 130, 520, "rec_turns"), (3, 100, 952, "rec_turns"),
                                          (2, 250, 1280, "rec_turns"), (2, 90, 2048, "rec_turns"),
                                          (3, 64, 1792, "rec_turns"), (2, 1024, 384, "rec_turns")])
def test_large_batches_match_oracle(T, B, d, kernel):
    """Without the flag: more groups than the device has CTAs for (the first case: a CTA for each, but more
    than the 64 rows the plans of rec_reg go up to); E1, E1 without a backward pass, and the state as its
    own gate (E33)."""
    inp = orc.make_e1_inputs(T, B, d, seed=d - B)
    with launches_of(kernel, 2):
        got, ref = run_compact(inp, 0)
    assert _lib.device_status()[0] == 0
    assert_close(errors(got, oracle_e1(ref)), TOL[torch.bfloat16], f"T{T} B{B} d{d}")
    dev, _ = round_inputs(inp, torch.bfloat16)
    h, out, _ = H.mamba_gated_elman_forward(False, dev["x"], dev["z"], dev["h0"], dev["W_x"], dev["W_h"],
                                            dev["b"])
    assert torch.equal(h, got["h"]) and torch.equal(out, got["output"])
    h, out, v = H.e33_self_gate_forward(True, dev["x"], dev["h0"], dev["W_x"], dev["W_h"], dev["b"])
    dx, dWx, dWh, db = H.e33_self_gate_backward(dev["W_x"], dev["W_h"], dev["x"], h, v, dev["d_output"])
    f = orc.e33_forward(ref["x"], ref["h0"], ref["W_x"], ref["W_h"], ref["b"])
    g = orc.e33_backward(ref["W_x"], ref["W_h"], ref["x"], f["h"], f["v"], ref["d_output"])
    assert_close(errors(dict(h=h, output=out, v=v, dx=dx, dW_x=dWx, dW_h=dWh, db=db), {**f, **g}),
                 TOL[torch.bfloat16], "self gate")


@pytest.mark.parametrize("T,B,d", [(2, 576, 256), (2, 640, 1280), (3, 256, 2048)])
def test_larger_batches_stay_with_the_tcgen05_kernel(T, B, d):
    """Over 512 rows, or six turns of 32 rows of W."""
    inp = orc.make_e1_inputs(T, B, d, seed=B)
    with launches_of("rec_tc", 2):
        got, ref = run_compact(inp, 0)
    assert _lib.device_status()[0] == 0
    assert_close(errors(got, oracle_e1(ref)), TOL[torch.bfloat16], f"T{T} B{B} d{d}")


def test_long_chain_agrees_with_one_group_per_set():
    """300 steps, many rounds of the ring and the buffers, against the kernel without turns."""
    inp = orc.make_e1_inputs(300, 29, 1280, seed=1)
    got, _ = run_compact(inp)
    other, _ = run_compact(inp, 0)
    for k in got:
        assert orc.rel_err(got[k].float().cpu(), other[k].float().cpu()) < 1e-2, k


def test_wait_that_runs_out_ends_the_launch():
    """Both directions: the launch returns, the status names the kernel, the next call is right."""
    inp = orc.make_e1_inputs(8, 24, 1280, seed=2)
    dev, ref = round_inputs(inp, torch.bfloat16)
    good, _ = run_compact(inp)
    _lib.device_status(clear=True)
    # the recurrences alone: the products around them have waits of their own
    for kid, call in (
            (2, lambda: H.e1_recurrence_forward(True, dev["x"], dev["z"], dev["h0"], dev["W_h"],
                                                H.FLAG_COMPACT)),
            (3, lambda: H.e1_recurrence_backward(dev["W_h"], dev["z"], good["h"], good["v"],
                                                 dev["d_output"], None, H.FLAG_COMPACT))):
        with option("spin_limit", 5000), option("test_stall_step", 4):
            call()
            torch.cuda.synchronize()
        code, detail = _lib.device_status()
        _lib.device_status(clear=True)
        assert code == 3 and (detail >> 24) & 0xFF == kid
    got, _ = run_compact(inp)
    assert_close(errors(got, oracle_e1(ref)), TOL[torch.bfloat16], "after the give-up")


def test_time_slots_of_2_gib_stay_with_the_kernel_that_counts_in_64_bits():
    """(No launch: what the planner says.)"""
    d = 136
    fits = (2 ** 30 - 1) // d
    assert H.recurrence_blocks(torch.bfloat16, 2, fits, d) > 0
    assert H.recurrence_blocks(torch.bfloat16, 2, fits + 1, d) == 0
