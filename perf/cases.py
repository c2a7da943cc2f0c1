"""Performance cases of the TTT operators: what a program that trains or serves a TTT layer calls.

A case is one call pattern of the public API at one size:

  op         "mlp" (two-layer inner model), "linear" (one-layer inner model) or "layer" (the MLP operator
             together with the token-layout, learning-rate-gate and output-norm kernels around it)
  mode       "fwd" (prefill / evaluation / the forward of a chunk) or "train" (forward and backward)
  B, H, NC   batch, heads, mini-batches of 64 tokens (sequence length / 64); head dimension 64
  cgs        checkpoint_group_size
  eta        scale of the learning-rate gate
  final      whether the state after the last mini-batch is asked for (sequences processed in chunks)

B * H is the number of independent (batch, head) streams, NC the length of each one's serial chain: together
they decide whether a call is bound by latency (few streams, short), by the chain (few streams, long) or by
throughput (more streams than the GPU has SMs).
"""
import math

import torch

from ttt_tk_b200.autograd import ttt_mlp
from ttt_tk_b200.buffers import GRAD_NAMES, alloc_backward_buffers, alloc_checkpoints
from ttt_tk_b200.glue import eta_gate, eta_gate_backward, pack_layernorm_backward, unpack_layernorm
from ttt_tk_b200.layout import pack_tokens, unpack_tokens
from ttt_tk_b200.ops import (linear_backward_scratch_bytes, ttt_backward, ttt_forward, ttt_linear_backward,
                             ttt_linear_forward)

BF16, F32 = torch.bfloat16, torch.float32
HEADS = (4, 12, 16, 24, 32)      # 256-, 768-, 1024-, 1536- and 2048-wide models


def _case(op, mode, B, H, NC, cgs, eta=0.1, final=False, name=None):
    c = {"op": op, "mode": mode, "B": B, "H": H, "NC": NC, "cgs": cgs, "eta": eta, "final": final}
    return dict(c, name=name) if name else c


def listed():
    return [
        # one mini-batch of one sequence, the state carried from call to call: the smallest call there is
        _case("mlp", "fwd", 1, 12, 1, 1, final=True, name="mlp fwd one mini-batch"),
        # training step of a toy model: one short sequence, four heads
        _case("mlp", "train", 1, 4, 32, 4, name="mlp train 4 streams"),
        # evaluation of a 768-wide model at 2048 tokens
        _case("mlp", "fwd", 4, 12, 32, 4, name="mlp fwd 48 streams"),
        # training step, odd batch and length, last checkpoint group incomplete
        _case("mlp", "train", 5, 12, 37, 5, name="mlp train 60 streams ragged"),
        # training step of a 2048-wide model at 8192 tokens: the ordinary large call
        _case("mlp", "train", 4, 32, 128, 8, name="mlp train 128 streams"),
        # long context: one sequence of 16384 tokens
        _case("mlp", "train", 1, 32, 256, 16, name="mlp train 16384 tokens"),
        # large-batch prefill of a 1536-wide model at 4096 tokens: the largest forward
        _case("mlp", "fwd", 64, 24, 64, 16, name="mlp fwd 1536 streams"),
        # the same calls with the one-layer inner model
        _case("linear", "fwd", 1, 12, 4, 4, final=True, name="linear fwd 4 mini-batches"),
        _case("linear", "train", 4, 32, 128, 8, name="linear train 128 streams"),
        _case("linear", "train", 13, 24, 37, 6, eta=1.0, name="linear train 312 streams ragged"),
        _case("linear", "fwd", 64, 24, 64, 16, name="linear fwd 1536 streams"),
        # a whole layer core from token-major activations and back, forward and backward
        _case("layer", "train", 4, 12, 32, 5, name="layer train 48 streams"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(("mlp", "mlp", "linear", "layer"))
    mode = "train" if op == "layer" else rng.choice(("fwd", "train"))
    most = 65536 if mode == "fwd" else 16384       # streams x mini-batches, below the largest listed case's
    H = rng.choice(HEADS)
    B = _log_int(rng, 1, 64)
    NC = _log_int(rng, 1, max(1, min(256, most // (B * H))))
    # from a checkpoint at every mini-batch to one per call; about sqrt(NC) is what callers use
    cgs = min(NC, max(1, int(round(math.sqrt(NC) * math.exp(rng.uniform(-0.7, 0.7))))))
    eta = rng.choice((0.01, 0.1, 1.0)) if NC <= 64 else 0.1
    return _case(op, mode, B, H, NC, cgs, eta, final=mode == "fwd" and op != "layer" and rng.random() < 0.5)


class _State:
    """The tensors a program has in hand before the call."""


def prepare(case, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    rn = lambda *s: torch.randn(*s, generator=g, dtype=F32, device="cuda")      # noqa: E731
    rb = lambda *s: torch.randn(*s, generator=g, dtype=BF16, device="cuda")     # noqa: E731
    new = lambda *s, dt=F32: torch.empty(*s, dtype=dt, device="cuda")           # noqa: E731
    B, H, NC, cgs = (case[k] for k in ("B", "H", "NC", "cgs"))
    s = _State()
    s.case = case
    s.gamma, s.beta = 1 + 0.02 * rn(1, H, 1, 64), 0.02 * rn(1, H, 1, 64)
    linear = case["op"] == "linear"
    if linear:
        s.init = [0.02 * rn(B, H, 64, 64), 0.02 * rn(B, H, 1, 64)]
    else:
        s.init = [0.02 * rn(B, H, 64, 256), 0.02 * rn(B, H, 1, 256), 0.02 * rn(B, H, 256, 64), 0.02 * rn(B, H, 1, 64)]

    if case["op"] == "layer":
        T, D = NC * 64, H * 64
        s.q, s.k, s.v, s.dy = (rb(B, T, D) for _ in range(4))
        s.logits = rb(B, T, H)
        s.out_gamma, s.out_beta = 1 + 0.02 * rn(D), 0.02 * rn(D)
        for t in (s.gamma, s.beta, *s.init):
            t.requires_grad_()
        return s

    tok = (B, H, NC, 64, 64)
    s.q, s.k, s.v = rb(*tok), rb(*tok), rb(*tok)
    s.last_eta = (case["eta"] * torch.sigmoid(rn(B, H, NC, 64)) / 64).to(BF16)
    s.out = new(*tok, dt=BF16)
    n = -(-NC // cgs)
    s.ckpt = [new(B, H, n, 64, 64), new(B, H, n, 1, 64)] if linear else alloc_checkpoints(B, H, NC, cgs)
    s.final = [torch.empty_like(t) for t in s.init] if case["final"] else None
    if case["mode"] == "train":
        s.d_out = rb(*tok)
        s.d_last = [1e-3 * torch.randn(t.shape, generator=g, dtype=F32, device="cuda") for t in s.init]
        if linear:
            s.scratch = new(linear_backward_scratch_bytes(B, H, cgs), dt=torch.uint8)
            s.grads = [new(B, H, 1, 64), new(B, H, 1, 64), *(torch.empty_like(t) for t in s.init),
                       new(B, H, NC, 64, dt=BF16), *(new(*tok, dt=BF16) for _ in range(3))]
        else:
            s.scratch, grads = alloc_backward_buffers(B, H, NC, cgs)
            s.grads = [grads[k] for k in GRAD_NAMES]
    return s


def _run_layer(s):
    c = s.case
    q, k, v = pack_tokens(s.q, s.k, s.v)
    eta = eta_gate(s.logits, c["eta"] / 64)
    leaves = [t.detach().requires_grad_() for t in (q, k, v, eta)]
    out, state = ttt_mlp(*leaves, s.gamma, s.beta, *s.init, checkpoint_group_size=c["cgs"])
    y, stats = unpack_layernorm(out.detach(), s.out_gamma, s.out_beta, return_stats=True)
    d_out, d_out_gamma, d_out_beta = pack_layernorm_backward(s.dy, out.detach(), s.out_gamma, stats)
    d_q, d_k, d_v, d_eta, *d_params = torch.autograd.grad(out, [*leaves, s.gamma, s.beta, *s.init], d_out)
    d_tokens = unpack_tokens(d_q, d_k, d_v)
    d_logits = eta_gate_backward(s.logits, d_eta, c["eta"] / 64)
    return [y, *d_tokens, d_logits, d_out_gamma, d_out_beta, *d_params, *(t.detach() for t in state)]


def run(s):
    if s.case["op"] == "layer":
        return _run_layer(s)
    cgs = s.case["cgs"]
    x = (s.q, s.k, s.v, s.last_eta, s.gamma, s.beta)
    linear = s.case["op"] == "linear"
    forward = ttt_linear_forward if linear else ttt_forward
    forward(*x, *s.init, *s.ckpt, s.out, cgs, final_state=s.final)
    outs = [s.out, *s.ckpt, *(s.final or ())]
    if s.case["mode"] == "train":
        if linear:
            ttt_linear_backward(*x, *s.ckpt, *s.d_last, s.d_out, *s.grads, cgs, scratch=s.scratch)
        else:
            eta5 = s.last_eta.unsqueeze(-1)
            ttt_backward(*x[:3], eta5, *x[4:], *s.ckpt, s.out, *s.scratch, *s.d_last, s.d_out, *s.grads, cgs)
        # the norm gradients come as one row per batch element; the caller adds them up
        outs += [g.sum(dim=0) for g in s.grads[:2]] + s.grads[2:]
    return outs


def work(case):
    B, H, NC, cgs = (case[k] for k in ("B", "H", "NC", "cgs"))
    streams, linear = B * H, case["op"] == "linear"
    tile = 64 * 64 * 2                                        # one bf16 mini-batch tile
    state = (64 * 64 + 64) * 4 if linear else (2 * 64 * 256 + 256 + 64) * 4
    per_mb = 4 * tile + 128                                   # Q, K, V, eta in; Out (or the normed output) out
    layer = case["op"] == "layer"
    # initial state in; checkpoints out (a layer keeps them to itself); final state out
    states = 1 + (0 if layer else -(-NC // cgs)) + (1 if case["final"] or layer else 0)
    unit = 2 * 64 * 64 * (64 if linear else 256)              # one product of a mini-batch
    # products of a mini-batch: the forward's, and in training those of the backward and of its recomputation
    # from the checkpoints
    products = 3 if linear else 7
    if case["mode"] == "train":
        products += 3 + 6 if linear else 7 + 15
        per_mb += 4 * tile + 128                              # dOut in; dQ, dK, dV, d_eta out
        states += 1 if layer else 2                           # dL/d(initial state) out, dL/d(last state) in
    return {"bytes": streams * (NC * per_mb + states * state), "flops": streams * NC * products * unit}


def tolerance(case):
    # bf16 operands and outputs, fp32 state and accumulation; gradients pass through about twice as many
    # bf16-rounded intermediates as the forward
    return {"rel": 1e-2} if case["mode"] == "fwd" else {"rel": 2e-2}
