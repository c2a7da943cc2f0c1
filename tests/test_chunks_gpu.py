"""A sequence in chunks of any length, down to a single mini-batch, with the CTAs per stream named: bit for bit one call, every
checkpoint (one before each mini-batch) and the final state included."""
import pytest
import torch

from oracle import ttt_mlp as orc
from test_streaming_gpu import STATE, forward
from ttt_tk_b200 import take_status

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cluster", [1, 2, 4])
@pytest.mark.parametrize("lengths", [(1, 2, 3, 4, 7), (5, 3), (16, 1)])
def test_chunks_of_the_forward_equal_one_call(cluster, lengths):
    NC = sum(lengths)
    t = {k: v.cuda() for k, v in orc.make_inputs(1, 3, NC, seed=NC, eta_scale=1.0).items()}
    s0 = [t[k] for k in STATE]
    want = forward(t, s0, 0, NC, 1, cluster)
    parts, lo, state = [], 0, s0
    for n in lengths:
        parts.append(forward(t, state, lo, lo + n, 1, cluster))
        lo, state = lo + n, list(parts[-1][2])
    torch.cuda.synchronize()
    assert take_status() == 0
    assert torch.equal(torch.cat([p[0] for p in parts], dim=2), want[0])
    for i, c in enumerate(want[1]):
        assert torch.equal(torch.cat([p[1][i] for p in parts], dim=2), c), i
    for a, b in zip(state, want[2]):
        assert torch.equal(a, b)
