"""Hand-over between the two groups of the MLP forward (csrc/ttt_fwd_sm100.cu), on a model of its barriers: every
interleaving of the chain group, the output group and their tensor-core work is walked through, and no group may write
what the other's products still read.  The steps are written out here; which barrier the chain group waits for before it
rewrites the bf16 W1, with which parity, and which barriers the output group's MMA5 commits to come from the source."""
import os
import re

SRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "ttt_tk_b200", "csrc", "ttt_fwd_sm100.cu")


def from_source(text):
    """(barrier, parity) of the wait before EPI4, and the barriers that MMA5's first / second 128-row block commits to."""
    epi4 = text[text.index("// ---- MMA4: W1^T +="):text.index("// ---- EPI4: bf16")]
    bar, parity = re.search(r"if \(it > 0\) wait_bar\((BAR_W1\w+|BAR_ACCB), (\w+)\);", epi4).groups()
    issue = re.search(r"auto issue_mma5 = .*?\};", text, re.S).group(0)
    commits = re.findall(r"if \(lead( && blk == 1)?\) umma_commit\(&bars\[(\w+)\]\)", issue)
    return (bar, parity), [[b for cond, b in commits if blk == 1 or not cond] for blk in (0, 1)]


def walk(epi4_wait, mma5_commits, NC=4):
    """Explore all interleavings.  Returns the violations found; a state in which nothing can run counts as one."""
    chain, out = [], []
    for i in range(NC):
        par, prev = i & 1, (i & 1) ^ 1
        chain += [("wait", "W2RDY", par)]
        chain += [("wait", "SREAD", prev)] * (i > 0)
        chain += [("mma", ("R W2b", "W W1", "W W2"), ["MMA4", "W2UPD"])]
        chain += [("wait", epi4_wait[0], {"par": par, "prev": prev}.get(epi4_wait[1], epi4_wait[1]))] * (i > 0)
        chain += [("wait", "MMA4", par), ("touch", "W W1b"), ("arrive", "W1RDY")]
        out += [("wait", "W2UPD", par), ("touch", "R W2"), ("touch", "W W2b"), ("arrive", "W2RDY")]
        out += [("wait", "W1RDY", par), ("touch", "R W1"), ("touch", "R W2"), ("arrive", "SREAD")]
        for blk in (0, 1):
            out += [("mma", ("R W1b",), mma5_commits[blk], i + 1), ("wait", "BAR_ACCB", blk)]
        out += [("mma", ("R W2b",), ["ZB"]), ("wait", "ZB", par)]
    prog, bad, seen = (chain, out), set(), set()
    copies = lambda pc: chain[:pc].count(("touch", "W W1b"))      # rewrites of the bf16 W1 so far
    # per agent: position, tensor work in flight (indices of its mma steps, in issue order); barriers: completions
    stack = [((0, 0), ((), ()), (("W2RDY", 1),))]            # W2RDY: the initial copy of W2
    while stack:
        state = stack.pop()
        if state in seen:
            continue
        seen.add(state)
        pc, flight, bars = state
        count = dict(bars)

        def clash(agent, access, others):                    # `others`: whose products in flight the access must not meet
            kind, what = access.split()
            for a in others:
                for j in flight[a]:
                    if any(o.split()[1] == what and "W" in (kind, o[0]) for o in prog[a][j][1]):
                        bad.add((agent, access, f"mma {j} of agent {a}"))

        moved = False
        for a in (0, 1):
            if flight[a]:                                    # the oldest product in flight completes
                moved = True
                c = dict(count)
                for b in prog[a][flight[a][0]][2]:
                    c[b] = c.get(b, 0) + 1
                fl = list(flight)
                fl[a] = flight[a][1:]
                stack.append((pc, tuple(fl), tuple(sorted(c.items()))))
            if pc[a] == len(prog[a]):
                continue
            step = prog[a][pc[a]]
            c, fl = dict(count), list(flight)
            if step[0] == "wait":                            # a wait on parity P passes when the phase under way has parity 1 - P
                if count.get(step[1], 0) % 2 == int(step[2]):
                    continue
            elif step[0] == "arrive":
                c[step[1]] = c.get(step[1], 0) + 1
            elif step[0] == "touch":
                clash(a, step[1], (0, 1))
            else:
                for access in step[1]:                       # products of one issuer run in order; the other's may overlap
                    clash(a, access, (1 - a,))
                if step[1] == ("R W1b",) and copies(pc[0]) != step[3]:
                    bad.add((a, "R W1b", f"copy {copies(pc[0])} instead of {step[3]}"))
                fl[a] = flight[a] + (pc[a],)
            moved = True
            p = list(pc)
            p[a] += 1
            stack.append((tuple(p), tuple(fl), tuple(sorted(c.items()))))
        if not moved and pc != (len(chain), len(out)):
            bad.add(("stuck", pc))
    return bad


def test_no_interleaving_of_the_two_groups_overwrites_an_operand():
    epi4_wait, commits = from_source(open(SRC).read())
    assert walk(epi4_wait, commits) == set()


def test_the_model_sees_a_barrier_completed_twice_per_mini_batch():
    """EPI4 on the barrier of both blocks, parity 1: passes at once while neither block's product has been issued."""
    bad = walk(("BAR_ACCB", 1), [["BAR_ACCB"], ["BAR_ACCB"]])
    assert any(b[1] == "W W1b" for b in bad)
