"""Scratch slots of the two-CTA backward, with slot_of and wait_slot as csrc/ttt_bwd_pair_sm100.cu has them: whatever the
sizes, the recompute never takes a slot whose content the sweep still has to read, and never waits for a step that needs its
own group's end.  (test_pair_order_cpu.py has the slots' addresses and their hand-over, at a few sizes.)"""
import pytest

import kernel_order as ko
from test_pair_order_cpu import source

SRC = source()
LAMBDAS = ("first_of", "size_of", "slot_of", "steps_before", "wait_slot")
BODY = [s for s in SRC.body("ttt_bwd_pair_kernel")[1]
        if s[0] == "lambda" and s[1] in LAMBDAS or s[0] == "decl" and s[2][0][0] == "nslots"]


class Need:
    """wait_slot's leaves: the number of steps it waits for."""
    def acquire(self, w, need):
        self.need = need

    def f___all_sync(self, w, m, v):
        return True


def functions(NC, cgs):
    leaf, sc = Need(), ko.Scope()
    w = ko.Walker(SRC, leaf)
    sc.v.update(NC=NC, cgs=cgs, nck=-(-NC // cgs))
    for s in BODY:
        w.do(s, sc)
    call = lambda name, *a: w.ev(("call", ("id", name), [("num", x) for x in a]), sc)       # noqa: E731

    def need(g, j):
        leaf.need = 0
        call("wait_slot", g, j)
        return leaf.need
    return call, need, sc.v["nslots"]


@pytest.mark.parametrize("cgs", [2, 3, 4, 5, 7, 8, 12, 16, 20, 33])
def test_no_slot_is_taken_before_it_has_been_read(cgs):
    assert len(BODY) == len(LAMBDAS) + 1
    for NC in list(range(cgs + 1, 4 * cgs + 2)) + [7 * cgs - 1]:
        call, need, nslots = functions(NC, cgs)
        read_at = {}                                     # slot -> the step after which its content is free
        steps = 0
        for g in range(-(-NC // cgs)):
            size = call("size_of", g)
            slots = [call("slot_of", g, j) for j in range(size)]
            for j, s in enumerate(slots):
                assert 0 <= s < nslots
                assert need(g, j) >= read_at.get(s, 0), (NC, g, j)
                assert need(g, j) <= steps               # a step of an earlier group: the sweep can reach it
            for j, s in enumerate(slots):
                read_at[s] = steps + size - j            # (the sweep goes from the last mini-batch to the first)
            steps += size
        assert steps == NC
