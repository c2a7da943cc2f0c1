"""Order of every access of the kernels with two groups of warps to a CTA (csrc/ttt_fwd_sm100.cu, ttt_linear_fwd_sm100.cu,
ttt_linear_bwd_sm100.cu) and of the TTT-Linear forward with one, from their sources: see kernel_order.py."""
import functools
import os

import pytest

import kernel_order as ko
from test_pair_order_cpu import CSRC, FILES

# source, kernel, warps, mini-batches, group size
CASES = [("ttt_fwd", "ttt_fwd_kernel", 16, 4, 2), ("ttt_linear_fwd", "ttt_linear_fwd_kernel", 8, 4, 2),
         ("ttt_linear_fwd", "ttt_linear_fwd_pair_kernel", 16, 4, 2), ("ttt_linear_bwd", "ttt_linear_bwd_kernel", 16, 5, 2),
         ("ttt_linear_bwd", "ttt_linear_bwd_kernel", 16, 3, 1), ("ttt_linear_bwd", "ttt_linear_bwd_kernel", 16, 3, 4)]


@functools.lru_cache(maxsize=None)
def run(name, kernel, warps, NC, cgs):
    def edit(text):
        if kernel == "ttt_linear_fwd_kernel" and "namespace pair {" in text:      # (its sibling has constants of the same names)
            i = text.index("namespace pair {")
            text = text[:i] + text[ko.closing(text, text.index("{", i)) + 1:]
        # the count of freed slots, a volatile word
        return text.replace("*freed = m;", "st_release_cluster(mapa(smem_u32(freed), 0), m);") \
            .replace("while (*freed < need)", "while (ok && ld_acquire_cluster(freed) < need)")
    src = ko.Source(*[os.path.join(CSRC, f) for f in FILES[:-1] + [name + "_sm100.cu"]], edit=edit)
    src.barriers = {v: k for k, v in src.names.items() if k.startswith("BAR_")}
    p = ko.Struct(H=1, NC=NC, cgs=cgs, nck=-(-NC // cgs), drop_load=-1, wait_limit_ns=0, scratch=ko.Ptr("g", 1 << 40, 1))
    for k in ("gamma beta W1 b1 W2 b2 W1c b1c W2c b2c W1f b1f W2f b2f W b Wc bc Wf bf gW_last gb_last gW gb d_gamma d_beta "
              "status").split():
        setattr(p, k, ko.Ptr("x", 100 << 40, 4))
    for k in ("eta", "out", "d_eta"):
        setattr(p, k, ko.Ptr("x", 100 << 40, 2))
    maps = {f"tm{k}": i for i, k in enumerate(["Q", "K", "V", "Out", "Go", "DQ", "DK", "DV"])}
    return ko.Run(src, kernel, dict(maps, p=p), {1: src.names.get("SLOT_BYTES", 0) * cgs}, 1, warps, skip=("wait_bar",))


@pytest.mark.parametrize("case", CASES)
def test_every_wait_ends_and_the_scratch_holds_what_was_stored(case):
    r = run(*case)
    assert r.problems == [] and r.provenance() == []


@pytest.mark.parametrize("case", CASES)
def test_no_two_accesses_are_unordered(case):
    assert run(*case).races() == []


@pytest.mark.parametrize("case", CASES)
def test_no_waiter_is_overtaken(case):
    assert run(*case).phases() == set()
