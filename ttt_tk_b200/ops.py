"""Host-side mirror of the reference's operator interface.

`ttt_forward` and `ttt_backward` take the same positional tensors, in the same order, as the
functions the reference's extension module exports (test_time_training.cpp:24-104;
launchers kernels/ttt/ttt.cu:594-611 and kernels/ttt_backward/ttt.cu:1451-1495) and return
the `Out` tensor like they do.  They validate like the reference's TORCH_CHECKs
(kernels/ttt/ttt.cu:621-630, kernels/ttt_backward/ttt.cu:1507-1760) -- on every call, and a
little more strictly -- raising RuntimeError, then hand raw device pointers to the C ABI
(include/ttt_mlp_b200.h): both in native code (csrc/ttt_host.cpp), since a short call is bound by
its host time.  torch is used only for device memory and the current stream.

Differences from the reference, all documented in the header:
  * calls are stream-ordered and do not synchronise;
  * backward overwrites grad_L_XQ/XK/XV/last_eta (the reference accumulates into zero-filled
    buffers) and never writes `Out`.
"""
from . import _lib
from .build import load_host


def _check(cond, msg):
    if not cond:
        raise RuntimeError(msg)


_HOST = None


def _host():
    global _HOST
    if _HOST is None:
        host = load_host()      # may build: before the library is loaded
        _lib.lib()
        _HOST = host
    return _HOST


def _flags(sync, cluster, lost_load=False):
    """Flag word of the C ABI: bit 0 synchronise, bit 1 the failure-path test hook, bits 8..11 the number
    of CTAs (1, 2 or 4) that share one stream (0 / None: chosen per call)."""
    cluster = 0 if cluster is None else int(cluster)
    _check(cluster in (0, 1, 2, 4), "cluster must be None, 1, 2 or 4")
    return (_lib.FLAG_SYNC if sync else 0) | (_lib.FLAG_TEST_LOST_LOAD if lost_load else 0) | (cluster << 8)


def ttt_forward(XQ, XK, XV, last_eta, ttt_norm_weight, ttt_norm_bias, W1, b1, W2, b2,
                W1_checkpoints, b1_checkpoints, W2_checkpoints, b2_checkpoints, Out,
                checkpoint_group_size, *, final_state=None, sync=False, cluster=None, _lost_load=False):
    """TTT-MLP forward over the whole sequence; writes `Out` and the state checkpoints.

    Positional arguments: exactly the reference's (kernels/ttt/ttt.cu:594-611).
    Keyword-only extras (not in the reference): `final_state` = (W1, b1, W2, b2) fp32 tensors
    that receive the state after the last mini-batch; `sync` blocks until the result is ready
    and raises on a device-side failure; `cluster` forces how many CTAs share one (batch, head)
    stream (1, 2 or 4; default: chosen from B*H, the length, the group size and the GPU's SM count).
    A sequence in chunks, each call's `final_state` the next one's initial state, agrees with one
    long call within rounding; with `cluster` named it has its bits.
    """
    _host().forward(XQ, XK, XV, last_eta, ttt_norm_weight, ttt_norm_bias, W1, b1, W2, b2, W1_checkpoints,
                    b1_checkpoints, W2_checkpoints, b2_checkpoints, Out, checkpoint_group_size, final_state,
                    _flags(sync, cluster, _lost_load))
    return Out


def ttt_linear_forward(XQ, XK, XV, last_eta, ttt_norm_weight, ttt_norm_bias, W1, b1,
                       W1_checkpoints, b1_checkpoints, Out, checkpoint_group_size, *,
                       final_state=None, sync=False, _lost_load=False):
    """TTT-Linear forward over the whole sequence: `ttt_forward` with the inner model reduced to one linear
    layer (W1 [B,H,64,64], b1 [B,H,1,64]; no W2 / b2); writes `Out` and the state checkpoints.  The reference
    has no counterpart (it ships the MLP operator only).  `final_state` = (W1, b1) fp32 tensors that receive
    the state after the last mini-batch."""
    _host().linear_forward(XQ, XK, XV, last_eta, ttt_norm_weight, ttt_norm_bias, W1, b1, W1_checkpoints, b1_checkpoints,
                           Out, checkpoint_group_size, final_state, _flags(sync, None, _lost_load))
    return Out


def ttt_linear_backward(XQ, XK, XV, last_eta, ttt_norm_weight, ttt_norm_bias, W1_checkpoints, b1_checkpoints,
                        grad_L_W1_last, grad_L_b1_last, grad_L_XQW_mini_batch, grad_L_ttt_norm_weight,
                        grad_L_ttt_norm_bias, grad_L_W1_init, grad_L_b1_init, grad_L_last_eta, grad_L_XQ, grad_L_XK,
                        grad_L_XV, checkpoint_group_size, *, scratch=None, sync=False, _lost_load=False):
    """TTT-Linear backward: gradients of `ttt_linear_forward` from its checkpoints.  Outputs (overwritten):
    norm gradients per batch element fp32 [B,H,1,64], dL/d(initial state) fp32 [B,H,64,64] / [B,H,1,64],
    grad_L_last_eta bf16 [B,H,NC,64] (or [..., 64, 1]), grad_L_XQ / XK / XV bf16 [B,H,NC,64,64].  `scratch`: a
    uint8 CUDA tensor of at least `linear_backward_scratch_bytes(B, H, checkpoint_group_size)` bytes (allocated
    here when not given).  The reference has no counterpart."""
    _host().linear_backward(XQ, XK, XV, last_eta, ttt_norm_weight, ttt_norm_bias, W1_checkpoints, b1_checkpoints,
                            grad_L_W1_last, grad_L_b1_last, grad_L_XQW_mini_batch, grad_L_ttt_norm_weight,
                            grad_L_ttt_norm_bias, grad_L_W1_init, grad_L_b1_init, grad_L_last_eta, grad_L_XQ, grad_L_XK,
                            grad_L_XV, checkpoint_group_size, scratch, _flags(sync, None, _lost_load))


def linear_backward_scratch_bytes(B, H, checkpoint_group_size):
    """Bytes of scratch `ttt_linear_backward` needs."""
    return int(_lib.lib().ttt_b200_linear_backward_scratch_bytes(int(B), int(H), int(checkpoint_group_size)))


def ttt_backward(XQ, XK, XV, last_eta, ttt_norm_weight, ttt_norm_bias,
                 W1_checkpoints, b1_checkpoints, W2_checkpoints, b2_checkpoints, Out,
                 W1_init_group, b1_init_group, W2_init_group, b2_init_group,
                 x_hat_ln_group, std_ln_group, X2_group, Z1_group, Z1_bar_group, X2_bar_group,
                 grad_l_wrt_Z2_group, grad_l_wrt_Z1_group, x_hat_fused_group, grad_x_hat_fused_group,
                 grad_output_fused_group, std_fused_group,
                 grad_L_W1_last, grad_L_b1_last, grad_L_W2_last, grad_L_b2_last, grad_L_XQW_mini_batch,
                 grad_L_ttt_norm_weight, grad_L_ttt_norm_bias, grad_L_W1_init, grad_L_b1_init,
                 grad_L_W2_init, grad_L_b2_init, grad_L_last_eta, grad_L_XQ, grad_L_XK, grad_L_XV,
                 checkpoint_group_size, *, sync=False, cluster=None, _lost_load=False):
    """TTT-MLP backward with per-checkpoint-group rematerialisation.

    Positional arguments: exactly the reference's 42 tensors + int
    (kernels/ttt_backward/ttt.cu:1451-1495).  grad_L_ttt_norm_weight / bias hold one row per
    batch element ([B, H, 1, 64]); the caller sums over dim 0 as with the reference
    (kernels/ttt_backward/matching.py:522-523).  `cluster` as in `ttt_forward`; chunks have the bits of one
    call with 1 or 4 named, or with 2 where every chunk is longer than a group of at least two mini-batches.
    """
    _host().backward(XQ, XK, XV, last_eta, ttt_norm_weight, ttt_norm_bias, W1_checkpoints, b1_checkpoints,
                     W2_checkpoints, b2_checkpoints, Out, W1_init_group, b1_init_group, W2_init_group, b2_init_group,
                     x_hat_ln_group, std_ln_group, X2_group, Z1_group, Z1_bar_group, X2_bar_group,
                     grad_l_wrt_Z2_group, grad_l_wrt_Z1_group, x_hat_fused_group, grad_x_hat_fused_group,
                     grad_output_fused_group, std_fused_group, grad_L_W1_last, grad_L_b1_last, grad_L_W2_last,
                     grad_L_b2_last, grad_L_XQW_mini_batch, grad_L_ttt_norm_weight, grad_L_ttt_norm_bias,
                     grad_L_W1_init, grad_L_b1_init, grad_L_W2_init, grad_L_b2_init, grad_L_last_eta, grad_L_XQ,
                     grad_L_XK, grad_L_XV, checkpoint_group_size, _flags(sync, cluster, _lost_load))
    return Out


def take_status():
    """0, or 3 if a kernel of this process gave up on a bounded wait since the last take."""
    return _lib.lib().ttt_b200_take_status()
