"""The backward that gives a stream two CTAs, one recomputing and one sweeping: against the oracle where its pipeline of
checkpoint groups can go wrong (no, one and several slots beyond the group's; last group incomplete, or of one mini-batch;
odd numbers of streams, whose last cluster holds one; the sizes at which the launcher turns to it).

Gate as for the other backward kernels: relative L2 <= 3e-2 for every gradient against the fp32 oracle."""
import pytest
import torch

from ttt_tk_b200 import _lib
from test_cluster_backward_gpu import GRAD_NAMES, TOL, check, inputs, oracle_backward, oracle_forward, run_backward

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,H,NC,cgs", [(1, 1, 4, 2), (1, 3, 5, 2), (1, 1, 10, 3), (2, 1, 13, 4), (1, 2, 16, 4), (3, 1, 23, 9),
                                        (1, 1, 36, 16), (1, 2, 72, 24), (1, 32, 64, 16)])
@pytest.mark.parametrize("eta_scale", [0.1, 1.0])
def test_pair_backward_matches_oracle(B, H, NC, cgs, eta_scale):
    d = inputs(B, H, NC, seed=NC, eta_scale=eta_scale)
    ck = oracle_forward(d, cgs)
    res = run_backward(d, ck, cgs, 2)
    check(res, oracle_backward(d, ck, cgs), TOL, "two CTAs per stream")
    again = run_backward(d, ck, cgs, 2)
    for k in GRAD_NAMES:
        assert torch.equal(res[k], again[k]), f"{k} differs between two runs"


@pytest.mark.parametrize("H", [1, 33, 66, 67, 74, 150])
def test_every_stream_count_matches_the_one_cta_kernel(H):
    """One or two streams to a cluster, a last cluster with one, more clusters than the device runs at once."""
    d = inputs(1, H, 9, seed=H)
    ck = oracle_forward(d, 4)
    check(run_backward(d, ck, 4, 2), run_backward(d, ck, 4, 1), 1e-2, f"{H} streams against one CTA per stream")


def test_calls_that_pipeline_groups_take_two_ctas():
    f = _lib.lib().ttt_b200_backward_ctas
    c4, c2 = (_lib.lib().ttt_b200_cluster_capacity(c, 1) for c in (4, 2))
    assert [f(c4, 12, 4, 0), f(c4, 11, 4, 0), f(c4, 64, 3, 0), f(c4 + 1, 1, 1, 0), f(c2 + 1, 64, 8, 0)] == [2, 4, 4, 2, 1]
    assert [f(c4, 64, 8, c << 8) for c in (1, 2, 4, 3)] == [1, 2, 4, -1]
    p = _lib.lib().ttt_b200_backward_pairs
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    assert [p(c4, 12, 4, 0), p(c4, 11, 4, 0), p(c2, 2, 1, 0), p(c2, 8, 8, 0), p(c2, 9, 8, 0), p(sms, 9, 8, 0), p(sms + 5, 9, 8, 0),
            p(sms + 5, 8, 8, 0), p(c4, 64, 8, 3 << 8)] == [c4, 0, 0, 0, c2, 0, 5, 0, -1]


@pytest.mark.parametrize("rest", [1, 2, 67, 74])
@pytest.mark.parametrize("NC,cgs", [(3, 2), (9, 4)])
def test_last_small_turn_runs_as_pairs(rest, NC, cgs):
    """Streams beyond a multiple of the SMs: a second launch, whose streams start where the first's end (heads differ)."""
    lib, sms = _lib.lib(), torch.cuda.get_device_properties(0).multi_processor_count
    H = sms + rest
    if rest > lib.ttt_b200_cluster_capacity(2, 1):
        pytest.skip("more streams than the device runs as pairs at once")
    assert [lib.ttt_b200_backward_tail(s, NC, cgs, 0) for s in (sms, H, 2 * sms, 2 * sms + rest)] == [0, rest, 0, rest]
    assert lib.ttt_b200_backward_tail(H, cgs, cgs, 0) == lib.ttt_b200_backward_tail(H, NC, 1, 0) == 0
    assert lib.ttt_b200_backward_tail(H, NC, cgs, 1 << 8) == 0
    d = inputs(1, H, NC, seed=rest)
    ck = oracle_forward(d, cgs)
    now, one, two = (run_backward(d, ck, cgs, c) for c in (None, 1, 2))
    for k in GRAD_NAMES:
        assert torch.equal(now[k][:, :sms], one[k][:, :sms]), f"{k} of the first launch"
        assert torch.equal(now[k][:, sms:], two[k][:, sms:]), f"{k} of the second"
