"""Order of every access of the two-CTA backward (csrc/ttt_bwd_pair_sm100.cu), from its source: see kernel_order.py."""
import functools
import os
import re

import pytest

import kernel_order as ko

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "ttt_tk_b200", "csrc")
FILES = ["sm100_ptx.cuh", "ttt_device.cuh", "ttt_cluster.cuh", "ttt_internal.h", "ttt_bwd_pair_sm100.cu"]
# the scratch tensors that the launcher hands over, and their bytes per mini-batch of a group
SCRATCH = {"X2_group": 32768, "Z1_group": 32768, "grad_l_wrt_Z1_group": 32768, "X2_bar_group": 32768, "Z1_bar_group": 32768,
           "W1_init_group": 65536, "W2_init_group": 65536, "x_hat_fused_group": 8192, "grad_l_wrt_Z2_group": 8192,
           "x_hat_ln_group": 8192, "b1_init_group": 1024, "std_ln_group": 256, "std_fused_group": 256, "b2_init_group": 256}
# mini-batches, group size, streams, streams to a cluster: no, one and two slots beyond the group's; a last group of one
# mini-batch, incomplete and whole; a cluster of two streams, and one whose second is missing
CASES = [(5, 2, 1, 1), (9, 4, 1, 1), (12, 4, 1, 1), (8, 3, 1, 1), (10, 8, 1, 1), (3, 2, 2, 2), (3, 2, 1, 2)]


def source(edit=lambda text: text):
    return ko.Source(*[os.path.join(CSRC, f) for f in FILES], edit=edit)


def walk(src, NC, cgs, streams=1, per=1):
    host = src.text[src.text.index("uint8_t* const w1 ="):src.text.index("p.gW1_last =")]
    p = ko.Struct(sc=[0] * len(SCRATCH), stride=[0] * len(SCRATCH), spare=[0] * len(SCRATCH))
    sc = ko.Scope()
    sc.v.update(p=p, a=ko.Struct(**{k: ko.Ptr("g", i + 1 << 40, 1) for i, k in enumerate(SCRATCH)}))
    for st in ko.Block(host).all()[1]:
        ko.Walker(src, None).do(st, sc)
    for k in "gamma beta W1c b1c W2c b2c gW1_last gb1_last gW2_last gb2_last d_gamma d_beta gW1 gb1 gW2 gb2 status".split():
        setattr(p, k, ko.Ptr("x", 0, 4))
    p.eta, p.d_eta = ko.Ptr("x", 100 << 40, 2), ko.Ptr("x", 0, 2)
    p.H, p.NC, p.cgs, p.nck, p.first, p.streams = streams, NC, cgs, -(-NC // cgs), 0, streams
    p.drop_load, p.wait_limit_ns = -1, 0
    maps = {f"tm{k}": i for i, k in enumerate(["Q", "K", "V", "Go", "DQ", "DK", "DV"])}
    return ko.Run(src, "ttt_bwd_pair_kernel", dict(maps, p=p, kStreams=per),
                  {i + 1: n * streams * cgs for i, n in enumerate(SCRATCH.values())}, 2 * per, 20)


@functools.lru_cache(maxsize=None)
def run(*case):
    return walk(source(), *case)


def place(r, key):
    """Shared-memory area of a race: the last of the role's offsets up to it."""
    if key[0] != "s":
        return key[0]
    offs = [(v, k) for k, v in r.src.names.items() if isinstance(v, int) and
            re.match("(OFF|%s)_" % ("S" if key[1] < r.ctas // 2 else "R"), k) and v <= key[2]]
    return max(offs)[1]


@pytest.mark.parametrize("case", CASES)
def test_every_wait_ends_and_the_scratch_holds_what_was_stored(case):
    r = run(*case)
    assert r.problems == [] and r.provenance() == []


@pytest.mark.parametrize("case", CASES)
def test_no_two_accesses_are_unordered(case):
    r = run(*case)
    assert [(place(r, x[0]), *x) for x in r.races()] == []


@pytest.mark.parametrize("case", CASES)
def test_no_waiter_is_overtaken(case):
    assert run(*case).phases() == set()


@pytest.mark.parametrize("now,then,NC,what", [
    ("{E_PART, kNo, kNo,", "{kNo, kNo, kNo,", 3, "races"),                              # a product that waits for less
    ("{SGZ1, E_X, C2,", "{SGZ1, kNo, C2,", 3, "races"),
    ("wait(F_ZG);", "", 3, "races"),                                                    # an epilogue
    ("need = steps_before(g - 1) + own + 1;", "need = steps_before(g - 1) + own;", 9, "races"),      # a slot taken early
    ("w2 + 3 * 65536 + BIG;", "w2 + 2 * 65536 + BIG;", 5, "provenance"),                # arrays that share a slot's place
    ("BGROUP + (g & 1)", "BGROUP", 5, "phases"),                                        # one barrier for all groups
])
def test_the_model_sees_a_mistake(now, then, NC, what):
    src = source(lambda text: text.replace(now, then))
    assert src.text != source().text
    assert getattr(walk(src, NC, 2 if NC == 3 else 4), what)()
