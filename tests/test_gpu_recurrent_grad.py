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


# the tensor-map kernel (16-bit states, head dims 128, 192, 256; above, where rows are many: one to three column tiles, of which the last may be partly
# empty): sequences shorter than, equal to
# and just beyond the 64 steps of its copies, initial states (the row of h_{-1} that is filled in), batches that do not fill a
# split evenly, and the GRU, whose first gate's deltas come from a buffer of their own
@pytest.mark.parametrize("function,B,T,N,D", [
    ("lstm", 3, 1, 2, 128), ("lstm", 5, 64, 1, 256), ("lstm", 2, 65, 2, 128), ("lstm", 9, 130, 1, 192),
    ("gru", 4, 1, 3, 128), ("gru", 7, 63, 1, 192), ("gru", 3, 129, 2, 256),
    ("slstm", 6, 66, 1, 128), ("elman", 5, 70, 2, 256), ("elman", 11, 2, 1, 128),
    ("elman", 3, 129, 2, 128), ("lstm", 10, 64, 1, 768), ("gru", 7, 129, 1, 768), ("lstm", 21, 65, 1, 512), ("slstm", 50, 70, 1, 320),
    ("lstm", 75, 9, 2, 128), ("gru", 40, 130, 2, 128),
])
def test_parameter_gradients_at_chunk_edges(cuda_device, function, B, T, N, D):
    Wx, R, b, s0 = make_inputs(function, B, T, N, D, seed=B * T + D, random_init=True)
    cot = torch.randn(s0.shape[0], B, T, N, D, generator=torch.Generator().manual_seed(11), dtype=torch.float64).to(torch.bfloat16).to(torch.float64)
    if function == "slstm":
        cot[3] = 0.0  # the stabiliser state has no cotangent in the closed-form backward
    got = run_native(function, Wx, R, b, s0, cot=cot)
    ref = run_oracle(function, Wx, R, b, s0, cot=cot)
    assert_parity(function, got, ref, tag=f"{function} B{B} T{T} N{N} D{D}", zero_init=False)
