"""The low-rank recurrence with both factors in registers (csrc/lowrank_reg.cuh) where its splits can
go wrong: ranks around the 16-row tiles and the 256-column K ranges, widths that leave CTAs or warps
partly filled, batches around the 8-row groups and one that goes through in several launches;
against the CPU oracle, with the bf16 tolerance of the other parity tests."""
import pytest
import torch

from _gpu_cases import E5W, TOL, assert_close, errors, launches_of, option, oracle_e5, round_inputs, run_e5
from elman_b200 import _lib
from elman_b200 import hasty_pytorch_lib as H
from oracle import elman_oracle as orc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T,B,d,r,slices", [
    (1, 1, 64, 1, 1), (5, 3, 72, 7, 1), (6, 9, 136, 16, 1), (4, 33, 264, 17, 1), (7, 8, 520, 130, 1), (3, 76, 768, 121, 1),
    (3, 128, 1536, 255, 1), (3, 40, 1032, 257, 1), (4, 5, 2048, 512, 1), (3, 200, 1536, 270, 2)])
def test_ragged_shapes_match_oracle(T, B, d, r, slices):
    inp = orc.make_e5_inputs(T, B, d, r, seed=d + r + B)
    with launches_of("lowrank_reg", 2 * slices):
        got, ref = run_e5(inp, torch.bfloat16)
    assert _lib.device_status()[0] == 0
    assert_close(errors(got, oracle_e5(ref)), TOL[torch.bfloat16], f"T{T} B{B} d{d} r{r}")


def test_compact_flag_takes_the_single_cluster_kernel():
    inp = orc.make_e5_inputs(6, 16, 256, 48, seed=11)
    dev, _ = round_inputs(inp, torch.bfloat16)
    w = [dev[k] for k in E5W]
    with launches_of("lowrank_reg", 2):
        a = H.pure_lowrank_elman_forward(True, dev["x"], dev["h0"], *w, dev["b"])
        ga = H.pure_lowrank_elman_backward_carry(*w, dev["x"], *a[0::2], dev["d_output"])
    with launches_of("lowrank_tc", 2):
        b = H.pure_lowrank_elman_forward(True, dev["x"], dev["h0"], *w, dev["b"], H.FLAG_COMPACT)
        gb = H.pure_lowrank_elman_backward_carry(*w, dev["x"], *a[0::2], dev["d_output"], None, H.FLAG_COMPACT)
    for x, y in zip(list(a) + ga, list(b) + gb):
        assert orc.rel_err(x.float().cpu(), y.float().cpu()) < 1e-2


@pytest.mark.parametrize("T,B,d,r", [(60, 40, 264, 40), (60, 9, 200, 130), (40, 36, 1536, 270)])
def test_rank_vector_keeps_the_bits_it_had_on_the_cuda_cores(T, B, d, r):
    """Error against 64 bits of what the recurrence feeds back, beside the kernel that keeps the rank vector
    in fp32.  Both round the state to bf16; rounding the vector as well adds 6 % (measured, and about what
    a second error of the size of a third adds to the first), two bf16 parts leave 2^-18.  Two orders of
    summation differ by 0.5 %."""
    inp = orc.make_e5_inputs(T, B, d, r, seed=d)
    f = {k: v.bfloat16().double().cuda() for k, v in inp.items()}
    got, _ = run_e5(inp, torch.bfloat16)
    with option("rec_reg", 1):
        cores, _ = run_e5(inp, torch.bfloat16)
    h, v = [f["h0"]], []
    pre = (f["x"] @ f["V_x"].T) @ f["U_x"].T + f["b"]
    for t in range(T):
        v.append(pre[t] + (h[-1] @ f["V_h"].T) @ f["U_h"].T)
        h.append(torch.tanh(v[-1]))
    gate = torch.nn.functional.silu((f["x"] @ f["V_z"].T) @ f["U_z"].T)
    dv, nxt = [], torch.zeros_like(f["h0"])
    for t in reversed(range(T)):
        nxt = (f["d_output"][t] * gate[t] + (nxt @ f["U_h"]) @ f["V_h"]) * (1 - h[t + 1] ** 2)
        dv.append(nxt)
    want = {"h": torch.stack(h), "v": torch.stack(v), "db": torch.stack(dv).sum((0, 1))}
    for k, slack in (("h", 1.02), ("v", 1.02), ("db", 1.3)):    # (db: one number per feature, noisier)
        new, old = (orc.rel_err(x[k].double(), want[k]) for x in (got, cores))
        assert new < slack * old, (k, new, old)


def test_rank_vectors_that_are_no_numbers_pass_through():
    """inf and NaN in a state reach every feature of their own sequence and no other one."""
    inp = orc.make_e5_inputs(3, 40, 136, 20, seed=4)
    inp["h0"][1, 5], inp["h0"][2, 7] = float("inf"), float("nan")
    got, _ = run_e5(inp, torch.bfloat16, training=False)
    with option("rec_reg", 1):
        cores, _ = run_e5(inp, torch.bfloat16, training=False)
    assert _lib.device_status()[0] == 0
    bad = got["h"][1:].isnan().flatten(2).any(2).any(0)
    assert bad[2] and not bad[0] and not bad[3:].any()
    assert torch.equal(got["h"].isnan(), cores["h"].isnan())
