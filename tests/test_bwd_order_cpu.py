"""Order of every access of the one-CTA backward (csrc/ttt_bwd_sm100.cu), from its source: see kernel_order.py."""
import functools
import os

import pytest

import kernel_order as ko
from test_pair_order_cpu import CSRC, FILES

SCRATCH = {"sc_W1": 65536, "sc_W2": 65536, "sc_Z1": 32768, "sc_X2": 32768, "sc_gZ1": 32768, "sc_Z1b": 32768, "sc_X2b": 32768,
           "sc_xhf": 8192, "sc_gof": 8192, "sc_gZ2": 8192, "sc_xhln": 8192}
CASES = [(3, 2), (3, 3), (2, 1)]      # mini-batches, group size


@functools.lru_cache(maxsize=None)
def run(NC, cgs):
    src = ko.Source(*[os.path.join(CSRC, f) for f in FILES[:-1] + ["ttt_bwd_sm100.cu"]])
    src.barriers = {v: k for k, v in src.names.items() if k.startswith("BAR_")}
    p = ko.Struct(H=1, NC=NC, cgs=cgs, nck=-(-NC // cgs), drop_load=-1, wait_limit_ns=0, w_stride=65536)
    for k in ("gamma beta W1c b1c W2c b2c gW1_last gb1_last gW2_last gb2_last d_gamma d_beta gW1 gb1 gW2 gb2 sc_sigf sc_sigln "
              "status").split():
        setattr(p, k, ko.Ptr("x", 100 << 40, 4))
    for k in ("eta", "d_eta"):
        setattr(p, k, ko.Ptr("x", 100 << 40, 2))
    for k in ("dXQ", "dXK", "dXV"):
        setattr(p, k, ko.Ptr("x", 100 << 40, 1))
    for i, k in enumerate(SCRATCH):
        setattr(p, k, ko.Ptr("g", i + 1 << 40, 1))
    maps = {f"tm{k}": i for i, k in enumerate(["Q", "K", "V", "Go", "DQ", "DK", "DV"])}
    return ko.Run(src, "ttt_bwd_kernel", dict(maps, p=p), {i + 1: n * cgs for i, n in enumerate(SCRATCH.values())}, 1, 8,
                  skip=("wait_bar", "skip_bar"))


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
