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


def test_tensor_memory_is_read_by_whole_warps():
    """A wait is left lane by lane.  Between it and a load from tensor memory the warp comes together: wait_mma, or done."""
    epilogues = KERNEL[KERNEL.index("for (int it = 0;"):KERNEL.index("reg_give")]
    last = None
    for token in re.findall(r"\b(wait|wait_mma|done|done_tmem|frag_ld|tmem_ld\w+)\(", epilogues):
        if token == "frag_ld" or token.startswith("tmem_ld"):
            assert last != "wait"
        else:
            last = token
