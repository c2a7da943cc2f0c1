"""Edges of the kernels that split a stream between two groups of warps (MLP forward and TTT-Linear forward: chain and
output; TTT-Linear backward: recompute of one checkpoint group beside the sweep of another), against the CPU oracles:
the first mini-batches, where a group still waits for nothing, checkpoints after every one or a ragged last group, one or
many checkpoint groups, and stream counts on both sides of the number of SMs."""
import pytest
import torch

import test_backward_gpu as bwd
import test_forward_gpu as mlp
import test_linear_backward_gpu as lbwd
import test_linear_forward_gpu as lfwd
from oracle import ttt_mlp as orc
from ttt_tk_b200 import take_status, ttt_forward
from ttt_tk_b200.buffers import alloc_checkpoints

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,H,NC,cgs", [(1, 1, 1, 1), (1, 2, 2, 1), (1, 1, 3, 2), (1, 3, 5, 2), (2, 74, 3, 2), (1, 149, 5, 1)])
def test_two_group_kernels_match_oracle(B, H, NC, cgs):
    d = orc.make_inputs(B, H, NC, seed=NC)
    ref = orc.ttt_forward(d["XQ"], d["XK"], d["XV"], d["last_eta"], d["ttt_norm_weight"], d["ttt_norm_bias"],
                          d["W1"], d["b1"], d["W2"], d["b2"], cgs)
    mlp.check(mlp.run_forward(d, cgs, final=True), ref,
              [("Out", mlp.TOL_OUT)] + [(k, mlp.TOL_STATE) for k in ("W1_checkpoints", "W2_checkpoints", "W1_final", "W2_final")])

    d = lbwd.make(B, H, NC, seed=NC + 1)
    ref_fwd, ref_bwd = lbwd.oracle(d, cgs)
    lfwd.check(lfwd.run(d, cgs), ref_fwd)
    lbwd.check(lbwd.run(d, cgs), ref_bwd)


@pytest.mark.parametrize("NC,cgs", [(3, 4), (9, 1), (9, 2), (13, 4)])
def test_linear_backward_group_edges(NC, cgs):
    """One group only, groups of one mini-batch, and a ragged last group after odd and even numbers of whole ones."""
    d = lbwd.make(1, 3, NC, seed=NC)
    _, ref = lbwd.oracle(d, cgs)
    lbwd.check(lbwd.run(d, cgs), ref)


@pytest.mark.parametrize("H,NC,cgs", [(34, 3, 2), (74, 1, 1), (75, 3, 2)])
def test_mlp_backward_between_the_cluster_sizes(H, NC, cgs):
    """The stream counts at which the backward turns from four CTAs per stream to two and from two to one."""
    d = orc.make_inputs(1, H, NC, seed=H, backward=True)
    ck = orc.ttt_forward(d["XQ"], d["XK"], d["XV"], d["last_eta"], d["ttt_norm_weight"], d["ttt_norm_bias"],
                         d["W1"], d["b1"], d["W2"], d["b2"], cgs)
    bwd.check(bwd.run_backward(d, ck, cgs), bwd.oracle_backward(d, ck, cgs))


@pytest.mark.parametrize("NC,cgs", [(96, 1), (97, 2)])
def test_mlp_forward_with_every_sm_storing_checkpoints(NC, cgs):
    """One stream on every SM, a checkpoint after every one or two mini-batches: the output groups fall behind their chains
    on the stores.  Every stream must come out bit for bit as from a call of its own, where nothing competes."""
    B = torch.cuda.get_device_properties(0).multi_processor_count
    t = {k: v.cuda() for k, v in orc.make_inputs(B, 1, NC, seed=NC).items()}

    def call(lo, hi):
        x = {k: v if k.startswith("ttt_norm") else v[lo:hi] for k, v in t.items()}
        ck, out = alloc_checkpoints(hi - lo, 1, NC, cgs), torch.empty_like(x["XQ"])
        ttt_forward(x["XQ"], x["XK"], x["XV"], x["last_eta"], x["ttt_norm_weight"], x["ttt_norm_bias"],
                    x["W1"], x["b1"], x["W2"], x["b2"], *ck, out, cgs, cluster=1)
        return [out, *ck]

    together = call(0, B)
    for b in range(B):
        for a, s in zip(together, call(b, b + 1)):
            assert torch.equal(a[b:b + 1], s), b
    assert take_status() == 0
