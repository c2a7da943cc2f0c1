"""Backward of more streams than the device runs as pairs at once, in two turns of them (csrc/ttt_bwd_pair_sm100.cu)."""
import pytest
import torch

from test_cluster_backward_gpu import TOL, check, inputs, oracle_backward, oracle_forward, run_backward
from ttt_tk_b200 import _lib
from ttt_tk_b200.buffers import GRAD_NAMES

pytestmark = pytest.mark.gpu


def test_which_calls_take_two_turns_of_pairs():
    lib = _lib.lib()
    tail, c2 = lib.ttt_b200_backward_tail, lib.ttt_b200_cluster_capacity(2, 1)
    most = max(n for n in range(c2 + 1, 149) if tail(n, 48, 8, 0))
    assert [tail(n, 48, 8, 0) for n in (c2, c2 + 1, most, most + 1)] == [0, c2 + 1, most, 0]
    assert [tail(most, nc, cgs, 0) for nc, cgs in ((47, 8), (59, 6), (60, 6), (100, 5))] == [0, 0, most, 0]
    assert tail(most, 48, 8, 1 << 8) == 0 and lib.ttt_b200_backward_pairs(most, 48, 8, 0) == most
    assert lib.ttt_b200_backward_ctas(most, 48, 8, 0) == 1


def test_two_turns_are_the_forced_form():
    """A last cluster with one stream, an incomplete last group."""
    H, NC, cgs = 75, 49, 8
    d = inputs(1, H, NC, seed=1)
    ck = oracle_forward(d, cgs)
    now, two = run_backward(d, ck, cgs, None), run_backward(d, ck, cgs, 2)
    for k in GRAD_NAMES:
        assert torch.equal(now[k], two[k]), k


@pytest.mark.parametrize("NC,cgs,ctas", [(16, 8, 2), (15, 8, 4), (14, 7, 4), (21, 7, 2)])
def test_two_long_groups_take_a_pair(NC, cgs, ctas):
    """Where four CTAs per stream would fit: the form it takes, against the oracle (3e-2: every gradient's gate)."""
    lib = _lib.lib()
    assert lib.ttt_b200_backward_ctas(lib.ttt_b200_cluster_capacity(4, 1), NC, cgs, 0) == ctas
    d = inputs(1, 3, NC, seed=2)
    ck = oracle_forward(d, cgs)
    now = run_backward(d, ck, cgs, None)
    check(now, oracle_backward(d, ck, cgs), TOL, "gradients")
    for k, t in run_backward(d, ck, cgs, ctas).items():
        if k in GRAD_NAMES:
            assert torch.equal(now[k], t), k
