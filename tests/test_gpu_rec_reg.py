"""The dense recurrence with W in registers (csrc/rec_reg.cuh) at the sizes where its splits can go
wrong: batches around the 8-row groups, widths that leave a CTA, a warp's K range or a block of 32
columns partly filled, the smallest and the widest matrix; against the CPU oracle, with the bf16
tolerance of the other parity tests."""
import pytest
import torch

from _gpu_cases import TOL, assert_close, errors, launches_of, option, oracle_e1, run_e1
from elman_b200 import _lib
from elman_b200 import hasty_pytorch_lib as H
from oracle import elman_oracle as orc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T,B,d", [(1, 1, 8), (5, 3, 24), (6, 9, 40), (7, 8, 72), (5, 7, 136),
                                   (4, 33, 248), (6, 17, 264), (5, 64, 520), (4, 37, 952),
                                   (3, 61, 1000), (3, 5, 2040), (3, 64, 1536)])
def test_ragged_shapes_match_oracle(T, B, d):
    inp = orc.make_e1_inputs(T, B, d, seed=7 * d + B)
    with launches_of("rec_reg", 2):
        got, ref = run_e1(inp, torch.bfloat16)
    assert _lib.device_status()[0] == 0
    assert_close(errors(got, oracle_e1(ref)), TOL[torch.bfloat16], f"T{T} B{B} d{d}")


@pytest.mark.parametrize("B,d", [(32, 256), (19, 200)])
def test_long_chain_agrees_with_the_other_kernels(B, d):
    """200 steps, many rounds of the input ring: against the TMEM kernel or the CUDA cores."""
    inp = orc.make_e1_inputs(200, B, d, seed=d)
    got, _ = run_e1(inp, torch.bfloat16)
    with option("rec_reg", 1):
        other, _ = run_e1(inp, torch.bfloat16)
    for k in got:
        assert orc.rel_err(got[k].float().cpu(), other[k].float().cpu()) < 1e-2, k


def test_unaligned_weights_take_another_kernel():
    """W 4 bytes off a 16-byte boundary: same result from a kernel that does not need it aligned."""
    inp = orc.make_e1_inputs(5, 4, 64, seed=3)
    dev = {k: v.to(torch.bfloat16).cuda() for k, v in inp.items()}
    flat = torch.empty(64 * 64 + 2, dtype=torch.bfloat16, device="cuda")
    W = flat[2:].view(64, 64).copy_(dev["W_h"])
    a = H.mamba_gated_elman_forward(True, dev["x"], dev["z"], dev["h0"], dev["W_x"], dev["W_h"], dev["b"])
    b = H.mamba_gated_elman_forward(True, dev["x"], dev["z"], dev["h0"], dev["W_x"], W, dev["b"])
    assert orc.rel_err(b[1].float().cpu(), a[1].float().cpu()) < 1e-2


def test_contexts_with_too_little_room_take_another_kernel():
    """Where the blocks that wait for one another cannot all be resident, nothing of the launch runs and
    the next kernel in line takes the call: dense in both precisions, low-rank, generation step."""
    from elman_b200.ladder_lm import LadderLM
    from _gpu_cases import oracle_e5, run_e5
    inp, low = orc.make_e1_inputs(4, 5, 136, seed=1), orc.make_e5_inputs(3, 40, 136, 20, seed=2)
    torch.manual_seed(3)
    lm = LadderLM(vocab_size=64, dim=64, depth=2, level=1).cuda().bfloat16().eval()
    tok = torch.tensor([[3]]).cuda()
    for limit in (0, 1):
        own = 2 if limit == 0 else 0
        with option("test_resident_blocks", limit):
            with launches_of("rec_reg", own):
                got, ref = run_e1(inp, torch.bfloat16)
            assert_close(errors(got, oracle_e1(ref)), TOL[torch.bfloat16], f"bf16, limit {limit}")
            with launches_of("rec_f32", own):
                got, ref = run_e1(inp, torch.float32)
            assert_close(errors(got, oracle_e1(ref)), TOL[torch.float32], f"fp32, limit {limit}")
            with launches_of("lowrank_reg", own):
                got, ref = run_e5(low, torch.bfloat16)
            assert_close(errors(got, oracle_e5(ref)), TOL[torch.bfloat16], f"low rank, limit {limit}")
            before = _lib.launch_count()
            with torch.no_grad():
                lm(tok)
            assert (_lib.launch_count() - before > 2) == (limit == 1)
    assert _lib.device_status()[0] == 0


def test_calls_on_two_streams_do_not_wait_for_each_others_blocks():
    """Two calls whose blocks do not fit on the device together, at the same time."""
    T, B, d = 40, 64, 952
    calls = []
    for seed in (1, 2):
        inp = orc.make_e1_inputs(T, B, d, seed=seed)
        dev = {k: v.to(torch.bfloat16).cuda() for k, v in inp.items()}
        args = (True, dev["x"], dev["z"], dev["h0"], dev["W_x"], dev["W_h"], dev["b"])
        calls.append((torch.cuda.Stream(), args, H.mamba_gated_elman_forward(*args)))
    assert 2 * H.recurrence_blocks(torch.bfloat16, T, B, d) > 148
    torch.cuda.synchronize()
    outs = [[], []]
    for _ in range(20):
        for i, (stream, args, _) in enumerate(calls):
            with torch.cuda.stream(stream):
                outs[i].append(H.mamba_gated_elman_forward(*args))
    torch.cuda.synchronize()
    assert _lib.device_status()[0] == 0
    for (_, _, want), got in zip(calls, outs):
        assert all(torch.equal(a, b) for g in got for a, b in zip(g, want))
