"""Backward of the output norm at the edges of its layout: tokens side by side in a CTA (few heads), warps left over, two head
groups to a warp, parameter gradients that are not 16-byte aligned."""
import pytest
import torch

from ttt_tk_b200 import _lib
from ttt_tk_b200.glue import pack_layernorm_backward, unpack_layernorm

pytestmark = pytest.mark.gpu


def make(B, NC, H):
    g = torch.Generator().manual_seed(H)
    x = torch.randn(B, H, NC, 64, 64, generator=g).to("cuda", torch.bfloat16)
    dy = torch.randn(B, NC * 64, H * 64, generator=g).to("cuda", torch.bfloat16)
    gamma = (1 + 0.1 * torch.randn(H * 64, generator=g)).cuda()
    return x, dy, gamma, torch.zeros_like(gamma)


def exact(x, dy, gamma):
    B, H, NC = x.shape[:3]
    v = x.double().reshape(B, H, NC * 64, 64).transpose(1, 2).reshape(B, NC * 64, H * 64).requires_grad_()
    gm, bt = gamma.double().requires_grad_(), torch.zeros_like(gamma, dtype=torch.float64).requires_grad_()
    y = torch.nn.functional.layer_norm(v, (H * 64,), gm, bt, 1e-6)
    dx, dg, db = torch.autograd.grad(y, (v, gm, bt), dy.double())
    return dx.reshape(B, NC, 64, H, 64).permute(0, 3, 1, 2, 4), dg, db


def rel(a, b):
    return float((a.double() - b).norm() / b.norm())


@pytest.mark.parametrize("H", [1, 4, 5, 9, 12, 16, 17, 20, 32, 33, 64])
def test_matches_fp64(H):
    """dx is rounded to bf16 once (2^-9 of each element); the fp32 sums run over 192 tokens."""
    x, dy, gamma, beta = make(3, 1, H)
    _, stats = unpack_layernorm(x, gamma, beta, return_stats=True)
    got = pack_layernorm_backward(dy, x, gamma, stats)
    want = exact(x, dy, gamma)
    assert rel(got[0], want[0]) <= 2 ** -8 and max(rel(a, b) for a, b in zip(got[1:], want[1:])) <= 1e-5


def test_parameter_gradients_at_an_odd_address():
    x, dy, gamma, beta = make(1, 2, 12)
    _, stats = unpack_layernorm(x, gamma, beta, return_stats=True)
    dx, buf = torch.empty_like(x), torch.zeros(2, 12 * 64 + 8, device="cuda")
    dg, db = buf[0, 1:769], buf[1, 3:771]
    _lib.call_on(x.device, "ttt_b200_pack_layernorm_backward", dy.data_ptr(), x.data_ptr(), gamma.data_ptr(), stats.data_ptr(),
                 dx.data_ptr(), dg.data_ptr(), db.data_ptr(), 1, 128, 12)
    want = exact(x, dy, gamma)
    assert rel(dg, want[1]) <= 1e-5 and rel(db, want[2]) <= 1e-5
    assert buf[0, 0] == buf[1, 2] == buf[0, 769] == buf[1, 771] == 0
