"""GPU: the dR kernels at the sizes where they can go wrong: head groups that N does not fill, row ranges that end inside a stage, batch
rows that start inside one, column tiles above head dim 256 of which the last is partly empty."""
import pytest
import torch

from tests.util import assert_parity, make_inputs, run_native, run_oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("function", ["lstm", "gru", "elman"])
@pytest.mark.parametrize("D,N", [(16, 1), (16, 9), (32, 3), (32, 5), (64, 1), (64, 5), (96, 4), (128, 2), (320, 1), (512, 1)])
@pytest.mark.parametrize("B,T,state_f32", [(1, 2, False), (5, 13, True), (3, 70, False)])
def test_recurrent_grad_edges(cuda_device, function, D, N, B, T, state_f32):
    Wx, R, b, s0 = make_inputs(function, B, T, N, D, seed=D + N + T, random_init=True, state_f32=state_f32)
    cot = torch.randn(s0.shape[0], B, T, N, D, generator=torch.Generator().manual_seed(T), dtype=torch.float64).to(torch.bfloat16).to(torch.float64)
    got = run_native(function, Wx, R, b, s0, cot=cot, state_f32=state_f32)
    ref = run_oracle(function, Wx, R, b, s0, cot=cot)
    assert_parity(function, got, ref, tag=f"{function} D{D} N{N} B{B} T{T}", zero_init=False)
