"""GPU: batches of more than 524 280 rows, where the time loops' 8-row tiles outnumber what a grid holds in y.  Rows never meet in the loops,
so the oracle runs the first and last of them; dR and db follow from the deltas (dWx) of all rows in fp64."""
import numpy as np
import pytest
import torch

from flashrnn_b200 import flashrnn
from tests.util import GRAD_REL_L2, H_MAX_ABS, cell_dims, max_abs, rel_l2, run_oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("function,B,D", [("lstm", 600001, 64), ("gru", 524281, 128), ("slstm", 600001, 64), ("lstm", 524281, 320)])
def test_more_rows_than_blocks_in_y(cuda_device, function, B, D):
    Gr, Gw, Gt, S = cell_dims(function)
    g = torch.Generator(device=cuda_device).manual_seed(B)
    randn = lambda *s: torch.randn(*s, generator=g, device=cuda_device)
    Wx = randn(B, 1, Gw, 1, D).bfloat16().requires_grad_(True)
    R = (randn(Gr, 1, D, D) / D ** 0.5).bfloat16().requires_grad_(True)
    b = (0.1 * randn(Gt, 1, D)).bfloat16().requires_grad_(True)
    s0 = 0.1 * randn(S, B, 1, 1, D)
    if function == "slstm":
        s0[2] = s0[2].abs() + 1.0
    s0 = s0.bfloat16().requires_grad_(True)
    states, _ = flashrnn(Wx, R, b, s0, function=function)
    dWx, dR, db, ds0 = torch.autograd.grad(states[0], (Wx, R, b, s0), torch.ones_like(states[0]))
    rows = torch.cat([torch.arange(8), torch.arange(B // 2, B // 2 + 8), torch.arange(B - 9, B)]).to(cuda_device)
    f = lambda t: t.detach().double().cpu()
    ref = run_oracle(function, f(Wx[rows]), f(R), f(b), f(s0[:, rows]))
    assert max_abs(f(states[0][rows]), ref["states"][0]) <= H_MAX_ABS
    assert rel_l2(f(dWx[rows]), ref["dWx"]) <= GRAD_REL_L2
    n = 3 if function == "slstm" else S
    assert rel_l2(f(ds0[:, rows])[:n], ref["ds0"][:n]) <= GRAD_REL_L2
    delta, h0 = dWx[:, 0, :, 0].double(), s0[0, :, 0, 0].double()  # [B,Gw,D], [B,D]
    shared = {0: 1, 1: 2} if function == "gru" else {i: i for i in range(Gw)}  # input gates whose delta is also the recurrent gate's
    for i, gate in shared.items():
        want = torch.einsum("bd,bp->dp", delta[:, i], h0)
        assert rel_l2(f(dR[gate, 0]), f(want)) <= GRAD_REL_L2
        assert rel_l2(f(db[gate, 0]), f(delta[:, i].sum(0))) <= GRAD_REL_L2
    assert np.isfinite(f(states.sum()).numpy())
