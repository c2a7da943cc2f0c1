"""Order of every access of the two-CTA forward (csrc/ttt_fwd_pair_sm100.cu), from its source: see kernel_order.py."""
import functools
import os

import pytest

import kernel_order as ko
from test_pair_order_cpu import CSRC, FILES

# mini-batches, group size, final state asked for, streams (two to a cluster, whose second may be missing)
CASES = [(1, 1, False, 1), (2, 1, True, 1), (5, 2, False, 1), (6, 4, True, 1), (3, 2, True, 2)]


class Agent(ko.Agent):
    def f_bulk_copy_peer(self, w, dst, src, nbytes, bar):
        """A bulk copy into another CTA's shared memory, which completes its bytes on a barrier there."""
        for d, s, n, b in self.each(w, dst, src, nbytes, bar):
            node = self.issue("copy to the other CTA")
            node.reads |= self.span(self.cta, s, n)
            node.writes |= self.span(dst.cta, d, n)
            self.r.loads.append(((bar.cta, (b - self.r.off_bar) // 8), n, node, None))


class NotNull(ko.Ptr):
    def __ne__(self, other):
        return True


def source(edit=lambda text: text):
    return ko.Source(*[os.path.join(CSRC, f) for f in FILES[:-1] + ["ttt_fwd_pair_sm100.cu"]], edit=edit)


def walk(src, NC, cgs, final, streams=1):
    p = ko.Struct(H=streams, NC=NC, cgs=cgs, nck=-(-NC // cgs), first=0, streams=streams, drop_load=-1, wait_limit_ns=0, eta=ko.Ptr("x", 100 << 40, 2))
    for k in "gamma beta W1 b1 W2 b2 W1c b1c W2c b2c b1f W2f b2f status".split():
        setattr(p, k, ko.Ptr("x", 100 << 40, 4))
    p.W1f = NotNull("x", 100 << 40, 4) if final else 0
    maps = {f"tm{k}": i for i, k in enumerate(["Q", "K", "V", "Out"])}
    plain, ko.Agent = ko.Agent, Agent
    try:
        return ko.Run(src, "ttt_fwd_pair_kernel", dict(maps, p=p), {}, 4, 20, vectors=src.names["OFF_SUM"])
    finally:
        ko.Agent = plain


@functools.lru_cache(maxsize=None)
def run(*case):
    return walk(source(), *case)


@pytest.mark.parametrize("case", CASES)
def test_every_wait_ends(case):
    assert run(*case).problems == []


@pytest.mark.parametrize("case", CASES)
def test_no_two_accesses_are_unordered(case):
    assert run(*case).races() == []


@pytest.mark.parametrize("case", CASES)
def test_no_waiter_is_overtaken(case):
    assert run(*case).phases() == set()


@pytest.mark.parametrize("now,then", [
    ("if (it > 0) wait(U_SENT);", ""),                                     # operands rewritten while they are copied
    ("if (it > 0 && !seen(X_FREE)) break;", ""),                           # sent into a buffer in use
    ("if (!seen(E_R) || !seen(OKT", "if (!seen(OKT"),                      # the state updated while a checkpoint is read
])
def test_the_model_sees_a_mistake(now, then):
    src = source(lambda text: text.replace(now, then))
    assert src.text != source().text
    r = walk(src, 5, 2, False)
    assert r.races() or r.phases() or r.problems
