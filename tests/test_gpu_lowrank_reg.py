"""The low-rank recurrence with both factors in registers (csrc/lowrank_reg.cuh) where its splits can
go wrong: ranks around the 16-row tiles and the 256-column K ranges, widths that leave CTAs or warps
partly filled, batches around the 8-row groups and batches that go through in several launches;
against the CPU oracle, with the bf16 tolerance of the other parity tests."""
import pytest
import torch

from _gpu_cases import E5W, TOL, assert_close, errors, oracle_e5, round_inputs, run_e5
from elman_b200 import _lib
from elman_b200 import hasty_pytorch_lib as H
from oracle import elman_oracle as orc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T,B,d,r", [(1, 1, 64, 1), (5, 3, 72, 7), (6, 9, 136, 16), (4, 33, 264, 17),
                                     (7, 8, 520, 130), (3, 76, 768, 121), (3, 128, 1536, 255),
                                     (3, 40, 1032, 257), (4, 5, 2048, 512)])
def test_ragged_shapes_match_oracle(T, B, d, r):
    inp = orc.make_e5_inputs(T, B, d, r, seed=d + r + B)
    before = _lib.tc_launch_count()
    got, ref = run_e5(inp, torch.bfloat16)
    assert _lib.tc_launch_count() - before >= 2
    assert _lib.device_status()[0] == 0
    assert_close(errors(got, oracle_e5(ref)), TOL[torch.bfloat16], f"T{T} B{B} d{d} r{r}")


def test_compact_flag_takes_the_single_cluster_kernel():
    inp = orc.make_e5_inputs(6, 16, 256, 48, seed=11)
    dev, _ = round_inputs(inp, torch.bfloat16)
    w = [dev[k] for k in E5W]
    a = H.pure_lowrank_elman_forward(True, dev["x"], dev["h0"], *w, dev["b"])
    b = H.pure_lowrank_elman_forward(True, dev["x"], dev["h0"], *w, dev["b"], H.FLAG_COMPACT)
    ga = H.pure_lowrank_elman_backward_carry(*w, dev["x"], *a[0::2], dev["d_output"])
    gb = H.pure_lowrank_elman_backward_carry(*w, dev["x"], *a[0::2], dev["d_output"], None, H.FLAG_COMPACT)
    for x, y in zip(list(a) + ga, list(b) + gb):
        assert orc.rel_err(x.float().cpu(), y.float().cpu()) < 1e-2
