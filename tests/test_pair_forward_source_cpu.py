"""What the two-CTA forward's source (csrc/ttt_fwd_pair_sm100.cu) promises outside of the order of accesses: how it ends, and
that warps are whole where an instruction needs them to be."""
import os
import re

from test_pair_order_cpu import CSRC

TEXT = re.sub(r"//.*", "", open(os.path.join(CSRC, "ttt_fwd_pair_sm100.cu")).read())
KERNEL = TEXT[TEXT.index("ttt_fwd_pair_kernel("):TEXT.index("int prepare_kernel()")]


def test_every_cta_of_a_cluster_meets_the_same_number_of_barriers():
    """A cluster holds two streams, and one may abort without the other: no barrier of the cluster stands in a branch."""
    depth, found = 0, []
    for token in re.findall(r"[{}]|cluster_(?:arrive|wait)\(\)", KERNEL[KERNEL.index("{"):]):
        depth += {"{": 1, "}": -1}.get(token, 0)
        if token not in "{}":
            found.append((token, depth))
    assert found == [("cluster_arrive()", 1), ("cluster_wait()", 1)] * 2
