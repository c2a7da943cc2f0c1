"""Backward of the output norm where a CTA takes fewer tokens side by side than its warps have room for: one to nine mini-batches
of one to seventeen heads."""
import pytest

from test_output_norm_backward_gpu import exact, make, pack_layernorm_backward, rel, unpack_layernorm

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,NC,H", [(1, 1, 1), (1, 1, 5), (1, 2, 2), (3, 1, 1), (1, 5, 3), (7, 1, 4), (1, 9, 1), (1, 1, 16), (1, 1, 17), (2, 1, 8)])
def test_matches_fp64(B, NC, H):
    """dx is rounded to bf16 once (2^-9 of each element); the fp32 sums run over at most 576 tokens."""
    x, dy, gamma, beta = make(B, NC, H)
    _, stats = unpack_layernorm(x, gamma, beta, return_stats=True)
    got = pack_layernorm_backward(dy, x, gamma, stats)
    want = exact(x, dy, gamma)
    assert rel(got[0], want[0]) <= 2 ** -8 and max(rel(a, b) for a, b in zip(got[1:], want[1:])) <= 1e-5
