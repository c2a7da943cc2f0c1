"""Order of every access of the kernels that split a stream's hidden units over a cluster (csrc/ttt_fwd_cluster_sm100.cu,
ttt_bwd_cluster_sm100.cu), from their sources: see kernel_order.py."""
import functools
import os
import re

import pytest

import kernel_order as ko
from test_pair_order_cpu import CSRC, FILES

# scratch of the backward.  x_hat_fused, x_hat_ln and dl/dZ2 are not followed: every CTA of a stream stores them, each reads
# back its own rows, or bits that all of them hold alike
SCRATCH = {"sc_W1": 65536, "sc_W2": 65536, "sc_Z1": 32768, "sc_X2": 32768, "sc_gZ1": 32768, "sc_Z1b": 32768, "sc_X2b": 32768}
CASES = [("fwd", 4, 3, 2), ("fwd", 2, 3, 2), ("bwd", 4, 2, 2), ("bwd", 4, 2, 1), ("bwd", 2, 3, 2)]      # kernel, CTAs, NC, cgs


def spelled_out(text):
    """What the reader of the sources does not know: names inside the configuration class, and the one store in PTX."""
    for now, then in (("typename C::RS ", "RS_object "), ("typename C::Sum ", "Sum_object "), ("C::RS::", "RS_"), ("RSx::", "RS_"),
                      ("C::Sum::", "Sum_"), ("C::", "C_"), (" RS::", " RS_"), (" Sum::", " Sum_"), ("do {", "{"), ("} while (0)", "}"),
                      ('_Pragma("unroll")', "")):
        text = text.replace(now, then)
    return re.sub(r'asm volatile\("st\.async\.weak[^:]*:[^"]*v4\.b32 .*?: "memory"\);', "st_async_f4(mapa(adr, peer), mapa(ba, peer));",
                  text, flags=re.S)


@functools.lru_cache(maxsize=None)
def run(which, ctas, NC, cgs):
    src = ko.Source(*[os.path.join(CSRC, f) for f in FILES[:-1] + [f"ttt_{which}_cluster_sm100.cu"]], edit=spelled_out)
    src.names["kC"] = ctas
    src.template("RowSplit", "RS_", kC=ctas, kExtras=which == "bwd")
    src.template("ClusterSum", "Sum_", kC=ctas, kSlotBytes_=18432 if which == "bwd" else 16384)
    c = src.template("Cfg", "C_", kC=ctas)
    src.barriers = {v: k for k, v in src.names.items() if k.startswith("BAR_")}
    p = ko.Struct(H=1, NC=NC, cgs=cgs, nck=-(-NC // cgs), drop_load=-1, wait_limit_ns=0)
    for k in ("gamma beta W1 b1 W2 b2 W1c b1c W2c b2c W1f b1f W2f b2f gW1_last gb1_last gW2_last gb2_last d_gamma d_beta gW1 gb1 gW2 "
              "gb2 sc_sigf sc_sigln status").split():
        setattr(p, k, ko.Ptr("x", 100 << 40, 4))
    for k in ("eta", "out", "d_eta", "dXQ", "dXK", "dXV"):
        setattr(p, k, ko.Ptr("x", 100 << 40, 2))
    for k in ("sc_xhf", "sc_gZ2", "sc_xhln"):
        setattr(p, k, ko.Ptr("x", 100 << 40, 1))
    for i, k in enumerate(SCRATCH):
        setattr(p, k, ko.Ptr("g", i + 1 << 40, 1))
    maps = {f"tm{k}": i for i, k in enumerate(["Q", "K", "V", "Out", "Go", "DQ", "DK", "DV"])}
    return ko.Run(src, f"ttt_{which}_cluster_kernel", dict(maps, p=p), {i + 1: n * cgs for i, n in enumerate(SCRATCH.values())},
                  ctas, 8, skip=("wait_bar", "skip_bar") if which == "bwd" else (), prefix="C_",
                  vectors=c["OFF_ETA"] if which == "fwd" else c["OFF_B2"])


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
