"""Scratch slots of the two-CTA backward (ttt_bwd_pair_sm100.cu: slot_of, wait_slot), restated: whatever the sizes, the
recompute never takes a slot whose content the sweep still has to read, and never waits for a step that needs its own
group's end."""
import pytest


@pytest.mark.parametrize("cgs", [2, 3, 4, 5, 7, 8, 12, 16, 20, 33])
def test_no_slot_is_taken_before_it_has_been_read(cgs):
    for NC in list(range(cgs + 1, 4 * cgs + 2)) + [7 * cgs - 1]:
        nck = -(-NC // cgs)
        nslots = cgs + cgs // 4
        size = lambda g: NC - (nck - 1) * cgs if g == 0 else cgs                              # noqa: E731
        before = lambda g: 0 if g == 0 else size(0) + (g - 1) * cgs                           # noqa: E731
        slot = lambda g, j: nslots - 1 - j if g & 1 else j                                    # noqa: E731

        def need(g, j):
            if g == 0:
                return 0
            own = j - (nslots - size(g - 1))
            if own >= 0:
                return before(g - 1) + own + 1
            return 0 if g == 1 or j >= size(g - 2) else before(g - 2) + size(g - 2) - j

        read_at = {}                                     # slot -> the step after which its content is free
        for g in range(nck):
            for j in range(size(g)):
                s = slot(g, j)
                assert 0 <= s < nslots
                assert need(g, j) >= read_at.get(s, 0), (NC, g, j)
                assert need(g, j) <= before(g)           # a step of an earlier group: the sweep can reach it
            for j in range(size(g)):
                read_at[slot(g, j)] = before(g) + size(g) - j
