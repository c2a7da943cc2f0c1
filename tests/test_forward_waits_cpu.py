"""Waits of the one-CTA MLP forward (csrc/ttt_fwd_sm100.cu): with any one of its hand-overs' waits or signals left out, the
order of accesses that kernel_order.py derives from the source shows it."""
import os
import re

import pytest

import kernel_order as ko
from test_pair_order_cpu import CSRC, FILES


def walk(edit, NC, cgs):
    src = ko.Source(*[os.path.join(CSRC, f) for f in FILES[:-1] + ["ttt_fwd_sm100.cu"]], edit=edit)
    src.barriers = {v: k for k, v in src.names.items() if k.startswith("BAR_")}
    p = ko.Struct(H=1, NC=NC, cgs=cgs, nck=-(-NC // cgs), drop_load=-1, wait_limit_ns=0, eta=ko.Ptr("x", 100 << 40, 2))
    for k in "gamma beta W1 b1 W2 b2 W1c b1c W2c b2c W1f b1f W2f b2f status".split():
        setattr(p, k, ko.Ptr("x", 100 << 40, 4))
    maps = {f"tm{k}": i for i, k in enumerate(["Q", "K", "V", "Out"])}
    return ko.Run(src, "ttt_fwd_kernel", dict(maps, p=p), {}, 1, 16, skip=("wait_bar",))


@pytest.mark.parametrize("NC,cgs", [(1, 1), (3, 1), (5, 3), (5, 2), (2, 2)])
def test_every_wait_ends_and_all_accesses_are_ordered(NC, cgs):
    r = walk(lambda text: text, NC, cgs)
    assert r.problems == [] and r.races() == [] and r.phases() == set()


WAITS = [
    "wait_bar(BAR_U2RDY, par);",                       # W2's update before U2 is there
    "wait_bar(BAR_R, par);",                           # the bf16 W2 rewritten under MMA3
    "if (it > 0) wait_bar(BAR_W2UPD, prev);",          # X2 rewritten under W2's update
    "if (it > 0) wait_bar(BAR_W1READ, prev);",         # the bf16 W1 rewritten under MMA5
    "if (it > 0) wait_bar(BAR_SREAD, prev);",          # the state updated while a checkpoint is read
    "wait_bar(BAR_W2RDY, par);",                       # MMA2 before the bf16 W2 is there
    "wait_bar(BAR_W1RDY, par);",                       # MMA5 before the bf16 W1 is there
]


@pytest.mark.parametrize("wait,cgs", [(w, c) for w in WAITS for c in (2, 3)])
def test_each_wait_is_needed(wait, cgs):
    seen = []
    r = walk(lambda text: seen.append(text.count(wait)) or text.replace(wait, ""), 5, cgs)
    assert sum(seen) == 1
    assert r.problems or r.races() or r.phases()


def test_loads_come_from_warps_that_issue_no_products():
    """The first warp of each 128-row block issues the chain group's products, the group's first warp the output group's."""
    text = open(os.path.join(CSRC, "ttt_fwd_sm100.cu")).read()
    chain, output = (int(n) // 32 for n in re.findall(r"const bool loader = gtid == (\d+);", text))
    assert "const bool issuer = quad == 0;" in text and chain % 4 != 0 and output != 0
