"""GPU: the float32 lane loops at the sizes where they can go wrong: head dims on both sides of every switch of their geometry, batches that
take 1, 2, 4 and 8 rows per CTA with a partial last tile, fewer steps than their input ring holds and one more."""
import pytest
import torch

from tests.test_gpu_float32 import _check
from tests.util import make_inputs, run_native, run_oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("function", ["lstm", "gru", "elman", "slstm"])
@pytest.mark.parametrize("D", [4, 20, 32, 36, 64, 72, 100, 128, 144, 256])
@pytest.mark.parametrize("B,T,N", [(1, 1, 1), (3, 5, 2), (41, 3, 13), (97, 2, 8)])
def test_float32_lane_loops_edges(cuda_device, function, D, B, T, N):
    Wx, R, b, s0 = make_inputs(function, B, T, N, D, seed=D + B, random_init=(function != "slstm"), dtype=torch.float32)
    cot = torch.randn(s0.shape[0], B, T, N, D, generator=torch.Generator().manual_seed(T), dtype=torch.float64).float().double()
    if function == "slstm":
        cot[1:] = 0
    clip = 0.05 if B == 3 else 0.0
    got = run_native(function, Wx, R, b, s0, cot=cot, dtype=torch.float32, **({"gradient_recurrent_clipval": clip} if clip else {}))
    ref = run_oracle(function, Wx, R, b, s0, cot=cot, clip=clip)
    _check(function, got, ref, f"{function} D{D} B{B} T{T} N{N}", n_ds0=1 if function == "slstm" else None)
