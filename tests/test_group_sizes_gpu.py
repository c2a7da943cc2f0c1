"""The forward's group size decides which states are stored, and nothing else: outputs, final state and the states that two sizes
both store are the same bits."""
import pytest
import torch

from test_cluster_forward_gpu import CK, FIN, nonzero_bias_inputs, run_forward

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cluster", [1, 2, 4])
@pytest.mark.parametrize("H,NC", [(3, 9), (150, 4)])
def test_groups_only_choose_what_is_stored(cluster, H, NC):
    d = nonzero_bias_inputs(1, H, NC, seed=NC, eta_scale=1.0)
    every = run_forward(d, 1, cluster)
    for cgs in (2, 3, NC):
        r = run_forward(d, cgs, cluster)
        for k in ["Out"] + FIN:
            assert torch.equal(r[k], every[k]), (cgs, k)
        for k in CK:
            assert torch.equal(r[k], every[k][:, :, ::cgs]), (cgs, k)
