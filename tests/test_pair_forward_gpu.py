"""The forward with two CTAs per stream (csrc/ttt_fwd_pair_sm100.cu): parity with the CPU oracle at the edges of its range,
and which calls take it."""
import pytest
import torch

from oracle import ttt_mlp as orc
from test_cluster_forward_gpu import CK, FIN, TOL, nonzero_bias_inputs, run_forward

pytestmark = pytest.mark.gpu


# the shortest, which only a caller asks for; a stream alone in its cluster; a checkpoint before every mini-batch, an incomplete last group, none but the first
@pytest.mark.parametrize("B,H,NC,cgs,eta", [(1, 1, 4, 4, 0.1), (1, 2, 7, 1, 1.0), (3, 1, 9, 4, 1.0), (1, 5, 16, 16, 0.1)])
def test_pair_forward_matches_oracle(B, H, NC, cgs, eta):
    d = nonzero_bias_inputs(B, H, NC, seed=NC, eta_scale=eta)
    ref = orc.ttt_forward(d["XQ"], d["XK"], d["XV"], d["last_eta"], d["ttt_norm_weight"], d["ttt_norm_bias"],
                          d["W1"], d["b1"], d["W2"], d["b2"], cgs)
    a, b = run_forward(d, cgs, 2), run_forward(d, cgs, 2)
    for k in ["Out"] + CK + FIN:
        assert torch.equal(a[k], b[k]), k
        assert orc.rel_l2(a[k], ref[k]) <= TOL, k


def test_calls_that_run_as_pairs():
    """Bit for bit the forced form, up to the streams that the device runs at once as pairs; one CTA each beyond."""
    from ttt_tk_b200 import _lib
    ctas = _lib.lib().ttt_b200_forward_ctas
    most = max(n for n in range(34, 75) if ctas(n, 6, 3, 0) == 2)
    assert [ctas(n, nc, cgs, 0) for n, nc, cgs in ((34, 5, 2), (34, 6, 1), (most, 6, 3), (most + 1, 6, 3))] == [1, 2, 2, 1]
    assert [ctas(12, nc, cgs, 0) for nc, cgs in ((1, 1), (15, 4), (16, 3), (16, 4))] == [4, 4, 4, 2]
    assert [ctas(12, 16, 4, n << 8) for n in (1, 2, 4, 3)] == [1, 2, 4, -1] and ctas(0, 16, 4, 0) == -1
    for n in (most, most + 1):
        d = nonzero_bias_inputs(1, n, 6, seed=n, eta_scale=1.0)
        out = {c: run_forward(d, 3, c)["Out"] for c in (None, 1, 2)}
        assert [torch.equal(out[c], out[None]) for c in (1, 2)] == [n > most, n <= most]
