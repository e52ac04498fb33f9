"""Work that users of flashrnn_b200 have it do, for timing one build of the package against another.

Three kinds of pass, each through the public entry points:

* ``train``: ``flashrnn(...)`` with gradients, then the backward pass of the layer's output h.  A layer on top of an LSTM or
  sLSTM sees ``states[0]`` only; GRU and Elman have no other state, so there the cotangent covers ``states`` as a whole.
* ``infer``: ``flashrnn(...)`` under ``torch.no_grad()`` (scoring, encoding, the prefill before decoding).
* ``step``:  one call of ``FlashRNNStepper.step`` (decoding; ``T`` is the chunk of tokens a call advances).

The inputs have the distributions of the benchmark configurations (``bench.py``): Wx ~ N(0,1), R ~ N(0,1/D), b ~ N(0,0.1)
(sLSTM: forget-gate bias in (3,6)), initial states zero or ~ N(0,0.1)."""
import math

import torch

from flashrnn_b200 import FlashRNNConfig, FlashRNNStepper, flashrnn

# recurrent gates, input gates, bias gates, states
DIMS = {"lstm": (4, 4, 4, 2), "gru": (3, 3, 4, 1), "elman": (1, 1, 1, 1), "slstm": (4, 4, 4, 4)}
TYPES = {"bfloat16": torch.bfloat16, "float16": torch.float16, "float32": torch.float32}


def _case(kind, cell, B, T, N, D, dtype="bfloat16", f32_states=False, init=False, clip=False):
    """``init``: the caller hands in initial states (and, training, takes their gradient); ``clip``: gradient clipping inside
    the recurrence (``gradient_recurrent_clipval``)."""
    return {"kind": kind, "cell": cell, "B": B, "T": T, "N": N, "D": D, "dtype": dtype, "f32_states": f32_states,
            "init": init, "clip": clip}


def listed():
    named = {
        # one token for a served batch, four heads of 256: a kernel of a few microseconds behind a host call
        "step_lstm_b16": _case("step", "lstm", 16, 1, 4, 256, init=True),
        # one token for one user, twelve heads of 64
        "step_gru_b1": _case("step", "gru", 1, 1, 12, 64, dtype="float16"),
        # prefill of a few prompts, odd batch and length
        "infer_slstm_b3": _case("infer", "slstm", 3, 777, 4, 192, f32_states=True),
        # encoding a large batch of sequences
        "infer_lstm_b256": _case("infer", "lstm", 256, 512, 12, 64, dtype="float16"),
        # the small float32 benchmark configuration: gradient checks, small models
        "train_lstm_f32": _case("train", "lstm", 4, 256, 2, 64, dtype="float32"),
        # the benchmark configurations of the four cells
        "train_lstm_b16": _case("train", "lstm", 16, 1024, 4, 256, init=True),
        "train_gru_b32": _case("train", "gru", 32, 2048, 8, 128),
        "train_slstm_b8": _case("train", "slstm", 8, 4096, 4, 192, f32_states=True),
        "train_elman_b1024": _case("train", "elman", 1024, 2048, 16, 64),
        # large-batch LSTM: throughput instead of latency
        "train_lstm_b1024": _case("train", "lstm", 1024, 512, 16, 64),
        # the top of the head-dim sweep: one head whose R does not fit the registers of its SMs
        "train_lstm_d768": _case("train", "lstm", 16, 1024, 1, 768),
        # a ragged last batch with gradient clipping, float16
        "train_gru_ragged": _case("train", "gru", 37, 333, 5, 96, dtype="float16", init=True, clip=True),
    }
    return [dict(c, name=n) for n, c in named.items()]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    while True:
        kind = rng.choice(["train", "train", "train", "infer", "step"])
        cell = rng.choice(list(DIMS))
        dtype = rng.choice(["bfloat16", "bfloat16", "bfloat16", "float16", "float32"])
        f32 = dtype == "float32"
        B, N = _log_int(rng, 1, 1024), _log_int(rng, 1, 24)
        T = _log_int(rng, 1, 16) if kind == "step" else _log_int(rng, 16, 1024 if f32 else 4096)
        D = rng.choice([20, 32, 64, 100, 128, 256] if f32 else [16, 32, 64, 64, 96, 128, 192, 256, rng.choice([384, 512, 768])])
        if N * D > 2048 or (D > 256 and T > 1024):
            continue
        # input elements, weighted by what one costs: long rows of R, and float32 outside the tensor cores
        load = B * T * N * D * DIMS[cell][1] * (32 if f32 else 16 if D > 256 else 4 if D > 64 else 1)
        if load <= 2 ** 31:
            return _case(kind, cell, B, T, N, D, dtype, f32 or rng.random() < 0.25, rng.random() < 0.5,
                         kind == "train" and rng.random() < 0.15)


def prepare(case, seed):
    Gr, Gw, Gt, S = DIMS[case["cell"]]
    B, T, N, D = case["B"], case["T"], case["N"], case["D"]
    dt = TYPES[case["dtype"]]
    sdt = torch.float32 if case["f32_states"] else dt
    g = torch.Generator(device="cuda").manual_seed(seed)

    def randn(*shape, dtype=dt):
        return torch.randn(*shape, generator=g, device="cuda", dtype=dtype)

    Wx = randn(B, T, Gw, N, D)
    R = (randn(Gr, N, D, D, dtype=torch.float32) / D ** 0.5).to(dt)
    b = 0.1 * randn(Gt, N, D, dtype=torch.float32)
    if case["cell"] == "slstm":
        b[1] = 3.0 + 3.0 * torch.rand(N, D, generator=g, device="cuda")
    b = b.to(dt)
    s0 = None
    if case["init"]:
        s0 = 0.1 * randn(S, B, 1, N, D, dtype=torch.float32)
        if case["cell"] == "slstm":
            s0[2] = s0[2].abs() + 1.0  # the normaliser of a running sequence
        s0 = s0.to(sdt)
    st = {"case": case, "Wx": Wx, "R": R, "b": b, "s0": s0}
    if case["kind"] == "step":
        st["stepper"] = FlashRNNStepper(R, b, function=case["cell"], batch_size=B, chunk=T, states=s0, dtype=case["dtype"],
                                        dtype_s="float32" if case["f32_states"] else None)
        return st
    st["call"] = {"function": case["cell"], "dtype": case["dtype"]}
    if case["clip"] or (case["f32_states"] and s0 is None):  # what the plain arguments cannot say
        st["call"] = {"config": FlashRNNConfig(
            function=case["cell"], head_dim=D, num_heads=N, batch_size=B, dtype=case["dtype"],
            dtype_s="float32" if case["f32_states"] else None, gradient_recurrent_clipval=0.5 if case["clip"] else None)}
    if case["kind"] == "train":
        st["leaves"] = [t.requires_grad_(True) for t in (Wx, R, b, s0) if t is not None]
        st["dout"] = randn(B, T, N, D, dtype=sdt) if S > 1 else randn(S, B, T, N, D, dtype=sdt)
    return st


def run(st):
    if st["case"]["kind"] == "step":
        out = st["stepper"].step(st["Wx"])
        return {"states": out, "carried": st["stepper"].states}
    if st["case"]["kind"] == "infer":
        with torch.no_grad():
            states, last = flashrnn(st["Wx"], st["R"], st["b"], st["s0"], **st["call"])
        return {"states": states, "last": last}
    states, last = flashrnn(st["Wx"], st["R"], st["b"], st["s0"], **st["call"])
    h = states[0] if states.shape[0] > 1 else states
    grads = torch.autograd.grad(h, st["leaves"], st["dout"])
    return {"states": states, "grads": list(grads)}


def work(case):
    Gr, Gw, Gt, S = DIMS[case["cell"]]
    E, N, D = case["B"] * case["T"] * case["N"] * case["D"], case["N"], case["D"]
    e = 4 if case["dtype"] == "float32" else 2
    es = 4 if case["f32_states"] else e
    params = (Gr * N * D * D + Gt * N * D) * e
    carried = S * case["B"] * N * D * es
    forward = Gw * E * e + params + S * E * es
    if case["kind"] == "step":
        return {"bytes": forward + 2 * carried, "flops": 2 * Gr * E * D}
    if case["init"]:
        forward += carried
    if case["kind"] == "infer":
        return {"bytes": forward, "flops": 2 * Gr * E * D}
    # cotangent of h in, gradients of Wx, R, b (and the initial states) out; three products: R h, R^T delta, delta h^T
    backward = E * es + Gw * E * e + params + (carried if case["init"] else 0)
    return {"bytes": forward + backward, "flops": 3 * 2 * Gr * E * D}


def tolerance(case):
    # float32: what the recurrence makes of reordered fp32 sums and another exp; 16-bit: roundings of h fed back T times
    return {"rel": 1e-4 if case["dtype"] == "float32" else 1e-2}
