"""GPU: the lane loops (head dims up to 256) at the sizes where they can go wrong: every head dim they are instantiated for, one
step, as many steps as and one more than their input ring holds (6), and batches around the 8-row tile; one CTA per head and
clusters, 8- and 16-row tiles.  The same for their forms for head dims above 256."""
import pytest
import torch

from tests.util import assert_parity, make_inputs, run_native, run_oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("function", ["lstm", "gru", "elman", "slstm"])
@pytest.mark.parametrize("D,cs,bt", [(16, 1, 8), (16, 1, 16), (32, 1, 16), (32, 2, 8), (64, 1, 8), (64, 1, 16), (64, 4, 16), (96, 3, 8), (96, 6, 16),
                                     (128, 2, 16), (128, 4, 8), (192, 6, 16), (256, 8, 8), (256, 8, 16)])
@pytest.mark.parametrize("B,T,state_f32", [(1, 1, False), (7, 6, True), (9, 7, False), (17, 2, True)])
def test_lane_loops_edges(cuda_device, function, D, cs, bt, B, T, state_f32):
    _check(function, 2, D, B, T, state_f32, cluster_size=cs, batch_tile=bt)


# 32, 48 and 64 units per CTA; R in registers alone, in shared memory too, and partly read from L2; with four heads the 16-row tiles
@pytest.mark.parametrize("function", ["lstm", "gru", "elman", "slstm"])
@pytest.mark.parametrize("N,D", [(1, 320), (4, 384), (1, 512), (4, 576), (1, 640), (1, 704), (1, 768), (4, 768), (1, 1024), (4, 1024)])
@pytest.mark.parametrize("B,T,state_f32", [(1, 1, False), (7, 6, True), (9, 5, False), (17, 2, True)])
def test_head_dims_above_256_edges(cuda_device, function, N, D, B, T, state_f32):
    _check(function, N, D, B, T, state_f32)


# the tiles the table picks, with the forms for 16-bit states where there are: few CTAs, and Elman's whole heads per CTA where CTAs fill the GPU
@pytest.mark.parametrize("function", ["lstm", "gru", "elman", "slstm"])
@pytest.mark.parametrize("N,D,B,T", [(2, 16, 9, 7), (1, 32, 9, 8), (3, 64, 1, 5), (2, 96, 9, 7), (1, 128, 17, 6), (1, 192, 9, 7), (32, 128, 33, 3), (19, 256, 57, 2)])
def test_lane_loops_own_tiles(cuda_device, function, N, D, B, T):
    _check(function, N, D, B, T, False)


# the clusters that large batches run with 16 rows
@pytest.mark.parametrize("function,D,cs", [("slstm", 96, 3), ("lstm", 96, 3), ("slstm", 128, 4), ("lstm", 128, 4), ("gru", 192, 6), ("gru", 256, 8)])
def test_lane_loops_16_rows(cuda_device, function, D, cs):
    _check(function, 2, D, 25, 8, function == "slstm", cluster_size=cs, batch_tile=16)


# head dim 16 with enough tiles for 16 rows in some of the loops
@pytest.mark.parametrize("function", ["lstm", "elman", "slstm"])
def test_head_dim_16_many_tiles(cuda_device, function):
    from flashrnn_b200 import _native

    N, B, T = 100, 233, 3
    plan = _native.query(_native.make_problem(function, B, T, N, 16, False, True))
    assert [_native.query_loop(plan, b).batch_rows for b in (False, True)] == [16, 16 if function == "elman" else 8]
    _check(function, N, 16, B, T, False)


# reverse loops with warps that only multiply, and the same head dims where there are more clusters than SMs for them: six, eight and ten warps
# beside each other, p tiles that divide among them and that do not, sums that stay in the CTA and that do not
@pytest.mark.parametrize("function,N,D,B,alone", [("lstm", 1, 96, 9, True), ("gru", 3, 96, 1, True), ("elman", 2, 96, 8, True), ("gru", 1, 128, 10, True),
                                                  ("slstm", 2, 128, 9, True), ("elman", 1, 128, 7, True), ("lstm", 3, 192, 9, True), ("gru", 2, 192, 3, True),
                                                  ("slstm", 1, 192, 17, True), ("elman", 1, 192, 9, True), ("lstm", 2, 256, 1, True), ("gru", 1, 256, 15, True),
                                                  ("slstm", 1, 256, 8, True), ("elman", 2, 256, 9, True), ("lstm", 23, 192, 3, True), ("slstm", 16, 256, 2, True),
                                                  ("gru", 46, 96, 2, True), ("gru", 34, 128, 3, False), ("gru", 23, 192, 2, False), ("elman", 34, 128, 1, False)])
def test_reverse_loops_with_multiplying_warps(cuda_device, function, N, D, B, alone):
    from flashrnn_b200 import _native

    few = _native.query_loop(_native.query(_native.make_problem(function, 8, 2, 1, D, False, True)), True).threads
    threads = _native.query_loop(_native.query(_native.make_problem(function, B, 2, N, D, False, True)), True).threads
    assert (threads == few) == alone
    _check(function, N, D, B, 5, function == "slstm" and B == 9)


# reverse loops that form dR themselves (T >= 24, sLSTM from 24 CTAs up) and their neighbours that do not: the last product with one and with two steps in it, rings of
# deltas and h at different places, ragged batches
@pytest.mark.parametrize("function,N,B", [("lstm", 2, 9), ("gru", 3, 15), ("slstm", 8, 17), ("gru", 1, 7), ("lstm", 1, 1), ("slstm", 23, 8)])
@pytest.mark.parametrize("T", [23, 24, 25, 26, 31])
def test_reverse_loops_that_form_dr(cuda_device, function, N, B, T):
    _check(function, N, 64, B, T, False)


# the same loops where every SM holds several of their CTAs: dR against the products of the very deltas and h it is formed of.  The returned dR is rounded to
# 8 bits; its fp32 sums are chains of at most T / 2 products of 16 rows and one addition per CTA of the head, each to 2^-22 of the sum of absolute values.
@pytest.mark.parametrize("function", ["lstm", "slstm"])
@pytest.mark.parametrize("T", [24, 33])
def test_loops_that_form_dr_on_a_full_gpu(cuda_device, function, T):
    from flashrnn_b200 import _native, flashrnn

    B, N, D = 1024, 16, 64
    assert _native.query_dr(_native.query(_native.make_problem(function, B, T, N, D, False, True)))[0]
    g = torch.Generator(device=cuda_device).manual_seed(T)
    randn = lambda *shape: torch.randn(*shape, generator=g, device=cuda_device, dtype=torch.bfloat16)
    Wx, R, b = randn(B, T, 4, N, D), randn(4, N, D, D) / D ** 0.5, randn(4, N, D) / 8
    leaves = [t.requires_grad_(True) for t in (Wx, R, b)]
    states, _ = flashrnn(*leaves, function=function)
    dWx, dR, _ = torch.autograd.grad(states[0], leaves, randn(B, T, N, D))
    h = torch.cat([torch.zeros_like(states[0][:, :1]), states[0].detach()[:, :-1]], 1)
    product = lambda x, y: torch.stack([torch.stack([x[:, :, q, n].reshape(-1, D).double().T @ y[:, :, n].reshape(-1, D).double() for n in range(N)]) for q in range(4)])
    want, size = product(dWx, h), product(dWx.abs(), h.abs())
    bound = 2.0 ** -8 * want.abs() + (T / 2 + 16 + B / 8) * 2.0 ** -22 * size + 2.0 ** -126
    assert bool(((dR.double() - want).abs() <= bound).all())


# enough clusters that Elman's forward loop takes CTAs of which two share an SM (R in registers alone, in shared memory too), and that the
# two loops split the head differently
@pytest.mark.parametrize("function,N,D", [("elman", 4, 512), ("elman", 3, 704), ("elman", 2, 1024), ("lstm", 5, 320), ("slstm", 5, 384)] +
                         # R in tensor memory: an odd number of k-pairs, with shared memory behind it, with L2 behind that, 8 and 16 rows
                         [("gru", 2, 576), ("lstm", 2, 832), ("gru", 1, 832), ("lstm", 1, 960), ("gru", 2, 960), ("slstm", 1, 704)])
def test_head_dims_above_256_many_clusters(cuda_device, function, N, D):
    _check(function, N, D, 147, 3, False)


# a tile the caller asks for: 64 units per CTA whatever the table says
@pytest.mark.parametrize("function,D,bt", [("lstm", 512, 16), ("gru", 384, 8), ("elman", 512, 16), ("slstm", 384, 16)])
def test_head_dims_above_256_forced_tile(cuda_device, function, D, bt):
    _check(function, 2, D, 17, 3, False, cluster_size=D // 64, batch_tile=bt)


def _check(function, N, D, B, T, state_f32, **tile):
    Wx, R, b, s0 = make_inputs(function, B, T, N, D, seed=D + T, random_init=True, state_f32=state_f32)
    S = s0.shape[0]
    cot = torch.randn(S, B, T, N, D, generator=torch.Generator().manual_seed(T), dtype=torch.float64).to(torch.bfloat16).to(torch.float64)
    if function == "slstm":
        cot[1:] = 0
    opts = dict(gradient_recurrent_clipval=0.05) if B == 9 else (dict(forward_clipval=0.5) if B == 7 else {})
    got = run_native(function, Wx, R, b, s0, cot=cot, state_f32=state_f32, **tile, **opts)
    ref = run_oracle(function, Wx, R, b, s0, cot=cot, clip=opts.get("gradient_recurrent_clipval", 0.0),
                     forward_clip=opts.get("forward_clipval", 0.0))
    assert_parity(function, got, ref, tag=f"{function} N{N} D{D} {tile} B{B} T{T}", zero_init=False)


# two clusters whose CTAs each take all of an SM's tensor memory must not share SMs: forward and reverse loops of both, on two streams at once
def test_head_dims_above_256_on_two_streams(cuda_device):
    from flashrnn_b200 import flashrnn

    calls = []
    for function, N, D in (("lstm", 4, 640), ("gru", 4, 768)):
        Wx, R, b, s0 = [t.to(cuda_device, torch.bfloat16) for t in make_inputs(function, 33, 24, N, D, seed=D)]
        calls.append((function, [Wx.requires_grad_(True), R, b, s0]))

    def passes(function, args):
        states, _ = flashrnn(*args, function=function)
        return states.detach(), torch.autograd.grad(states[0], args[0], torch.ones_like(states[0]))[0]

    alone = [passes(*c) for c in calls]
    streams = [torch.cuda.Stream(cuda_device) for _ in calls]
    torch.cuda.synchronize()
    together = []
    for _ in range(5):
        for stream, c in zip(streams, calls):
            with torch.cuda.stream(stream):
                together.append(passes(*c))
    torch.cuda.synchronize()
    for i, got in enumerate(together):
        assert all(torch.equal(x, y) for x, y in zip(got, alone[i % 2]))
