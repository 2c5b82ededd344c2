"""The single-precision kernels (csrc/rec_f32.cu, csrc/gemm_f32.cu) at the edges of their tiles: rows
and K ranges partly filled, batches around the 4-row groups and over one launch, products whose K is
cut over a cluster.  Tolerances: the parity tests' 1e-4 for a cell against the fp32 CPU oracle; 1e-6
for a product against fp64 (a sum of K terms is off by about sqrt(K) 2^-24, 2.4e-6 / 2 at K = 1600)."""
import pytest
import torch

from _gpu_cases import TOL, assert_close, errors, launches_of, option, oracle_e1, round_inputs, run_e1
from elman_b200 import _lib
from elman_b200 import hasty_pytorch_lib as H
from oracle import elman_oracle as orc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T,B,d,slices", [(1, 1, 8, 1), (7, 5, 12, 1), (5, 4, 184, 1), (6, 17, 260, 1), (4, 3, 516, 1),
                                          (3, 33, 1000, 3), (3, 2, 1024, 1)])
def test_recurrence_matches_oracle(T, B, d, slices):
    inp = orc.make_e1_inputs(T, B, d, seed=d + B)
    with launches_of("rec_f32", 2 * slices):
        got, ref = run_e1(inp, torch.float32)
    assert _lib.device_status()[0] == 0
    assert_close(errors(got, oracle_e1(ref)), TOL[torch.float32], f"fp32 T{T} B{B} d{d}")
    with option("rec_reg", 1):      # the cooperative kernel: the same arithmetic in another order
        other, _ = run_e1(inp, torch.float32)
    assert_close({k: orc.rel_err(got[k].cpu(), other[k].cpu()) for k in got}, 1e-5, "vs cooperative")


@pytest.mark.parametrize("op", [H.GEMM_NT, H.GEMM_NN, H.GEMM_TN])
@pytest.mark.parametrize("M,N,K", [(1, 1, 1), (64, 64, 16), (65, 67, 130), (44, 52, 1600), (300, 130, 260),
                                   (512, 256, 256)])
def test_products_of_every_form(op, M, N, K):
    g = torch.Generator().manual_seed(M + N + K)
    A = torch.randn(*((K, M) if op == H.GEMM_TN else (M, K)), generator=g)
    B = torch.randn(*((N, K) if op == H.GEMM_NT else (K, N)), generator=g)
    want = (A.double().T if op == H.GEMM_TN else A.double()) @ (B.double().T if op == H.GEMM_NT else B.double())
    bias = torch.randn(N, generator=g) if op == H.GEMM_NT else None
    out = H.gemm(op, A.cuda(), B.cuda(), None if bias is None else bias.cuda())
    base = want if bias is None else want + bias.double()
    assert orc.rel_err(out.double().cpu(), base) < 1e-6
    out = H.gemm(op, A.cuda(), B.cuda(), out=out, accumulate=True)
    assert orc.rel_err(out.double().cpu(), base + want) < 1e-6


def test_recurrence_gives_up_when_a_block_stalls_and_recovers():
    inp = orc.make_e1_inputs(8, 6, 260, seed=9)
    dev, ref = round_inputs(inp, torch.float32)
    good, _ = run_e1(inp, torch.float32)
    _lib.device_status(clear=True)
    for call in (lambda: H.e1_recurrence_forward(True, dev["x"], dev["z"], dev["h0"], dev["W_h"]),
                 lambda: H.e1_recurrence_backward(dev["W_h"], dev["z"], good["h"], good["v"], dev["d_output"])):
        with option("spin_limit", 5000), option("test_stall_step", 4):
            call()
            torch.cuda.synchronize()
        code, detail = _lib.device_status(clear=True)
        assert code == 3 and detail >> 24 == 1 and detail & 0xFFFFFF in (4, 5)   # the block, or one behind it
    got, _ = run_e1(inp, torch.float32)
    assert_close(errors(got, oracle_e1(ref)), TOL[torch.float32], "after the give-up")
