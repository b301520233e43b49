"""The barrier protocol of the gathering attention kernels, explored state by state on the CPU.

The kernels (mla_bf16.cuh, attn_fp8.cu) pass every item's Q and K / V blocks through a ring of slots;
their warps wait on mbarriers by PARITY, which answers for the right phase only while a waiter is at
most one phase behind.  Here one CTA of such a kernel is a set of agents -- two gather warps, QK^T
issue, PV issue, two softmax groups, epilogue -- that advance in every possible order; a test of a
barrier is the same parity comparison the hardware makes.  Ring depth, Q entries per item and the
depths of the barrier arrays are read from the sources."""
import itertools
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "litetopk_b200" / "csrc"


def _constants(source):
    src = (CSRC / source).read_text()

    def depth(name):      # entries of a barrier array of Misc, 1 for a single barrier
        m = re.search(r"uint64_t\s[^;]*\b%s(?:\[(\d+)\])?[;,]" % name, src)
        return int(m.group(1) or 1)

    ring = dict(slots=int(re.search(r"kSlots = (\d+)", src).group(1)), q_taken=depth("q_taken"),
                epi_ready=depth("epi_ready"))
    m = re.search(r"kQEntries = (\d+)", src)
    ring["q_entries"] = int(m.group(1)) if m else 1
    # a gather warp that did not request the Q entries itself may go by q_taken instead of slot_free
    ring["by_q_taken"] = "q_held" in src
    return ring


def _explore(blocks, slots, q_entries, q_taken, epi_ready, by_q_taken):
    """Every order of the agents' steps over items of ``blocks`` key blocks: the set of faults found
    ("overwrite": a copy into a slot whose last entry is still needed, "stuck": no agent can go on)."""
    n, first = len(blocks), [0]
    for b in blocks:
        first.append(first[-1] + b)
    nb = first[-1]
    item = [i for i, b in enumerate(blocks) for _ in range(b)]
    entry = [kb + q_entries * (item[kb] + 1) for kb in range(nb)]
    q_entry = [first[i] + q_entries * i for i in range(n)]
    kind = {e: ("K", kb) for kb, e in enumerate(entry)}
    kind.update({q_entry[i] + e: ("Q", i) for i in range(n) for e in range(q_entries)})
    soft = [[], []]       # softmax group: read S, publish P of its blocks; at an item's end wait, then arrive
    for i in range(n):
        for kb in range(first[i], first[i + 1]):
            soft[kb & 1] += [("S", kb), ("P", kb)]
        for g in (0, 1):
            soft[g] += [("wait", i), ("arrive", i)]
    at = [{x: j for j, x in enumerate(soft[g])} for g in (0, 1)]
    epi = [("Q", 0)]      # epilogue: move Q in, wait for the row scales, write O out
    for i in range(n):
        epi += ([("Q", i + 1)] if i + 1 < n else []) + [("scales", i), ("O", i)]
    q_moved = [sum(x[0] == "Q" for x in epi[:j]) for j in range(len(epi) + 1)]
    o_read = [sum(x[0] == "O" for x in epi[:j]) for j in range(len(epi) + 1)]

    def passes(completed, phase):               # mbarrier.try_wait.parity
        return (completed & 1) != (phase & 1)

    def nth(count, of, depth):                  # completions, among the first `count`, of the barrier item / block `of` uses
        return sum(1 for j in range(count) if j % depth == of % depth)

    faults, seen, stack = set(), set(), [(0,) * 10]
    while stack:
        st = stack.pop()
        if st in seen:
            continue
        seen.add(st)
        k0, v0, rq, k1, v1, qk, pv, s0, s1, ep = st
        s, moved = (s0, s1), q_moved[ep]
        nxt = []

        def go(**kw):
            nxt.append(tuple(kw.get(f, x) for f, x in zip(("k0", "v0", "rq", "k1", "v1", "qk", "pv", "s0", "s1", "ep"), st)))

        def freed(slot):                        # phases slot_free[slot] has completed
            return sum(1 for kb in range(pv) if entry[kb] % slots == slot) + \
                sum(1 for i in range(moved) for e in range(q_entries) if (q_entry[i] + e) % slots == slot)

        def live(e):                            # an older entry of e's slot is still needed
            while e >= slots:
                e -= slots
                what, x = kind[e]
                if x >= (pv if what == "K" else moved):
                    return True
            return False

        def done(x, g):
            return s[g] > at[g][x]

        def scales(i):                          # completions of the epi_ready barrier item i uses
            return sum(1 for j in range(i % epi_ready, n, epi_ready) if done(("arrive", j), 0) and done(("arrive", j), 1))

        for w, (k, v) in enumerate(((k0, v0), (k1, v1))):
            if v < k and passes(nth(qk, v, 8), v >> 3):
                go(**{"v%d" % w: v + 1})
            if k == nb:
                continue
            i = item[k]
            if w == 0 and rq < q_entries * (i + 1):                     # this warp requests Q first
                e = q_entry[i] + rq - q_entries * i
                if (e < slots or passes(freed(e % slots), e // slots - 1)) and \
                        (i == 0 or passes(nth(moved, i - 1, q_taken), (i - 1) // q_taken)):
                    if live(e):
                        faults.add("overwrite")
                    else:
                        go(rq=rq + 1)
                continue
            e = entry[k]
            if e >= slots and by_q_taken and kind[e - slots][0] == "Q":
                j = kind[e - slots][1]
                ok = passes(nth(moved, j, q_taken), j // q_taken)
            else:
                ok = e < slots or passes(freed(e % slots), e // slots - 1)
            if ok and live(e):
                faults.add("overwrite")
            elif ok:
                go(**{"k%d" % w: k + 1})
        if qk < min(k0, k1) and (qk > first[item[qk]] or moved > item[qk]) and (qk < 2 or done(("S", qk - 2), qk & 1)):
            go(qk=qk + 1)
        if pv < min(v0, v1) and done(("P", pv), pv & 1) and (pv > first[item[pv]] or o_read[ep] >= item[pv]):
            go(pv=pv + 1)
        for g in (0, 1):
            if s[g] == len(soft[g]):
                continue
            what, x = soft[g][s[g]]
            if what == "S":
                ok = qk > x and (x == first[item[x]] or done(("S", x - 1), g ^ 1))
            elif what == "P":
                ok = x < 2 or passes(nth(pv, x - 2, 4), (x - 2) >> 2)
            elif what == "wait":
                ok = x == 0 or passes(scales(x - 1), (x - 1) // epi_ready)
            else:
                ok = done(("wait", x), 0) and done(("wait", x), 1)
            if ok:
                go(**{"s%d" % g: s[g] + 1})
        if ep < len(epi):
            what, x = epi[ep]
            if what == "Q":
                ok = (x == 0 or qk >= first[x]) and rq >= q_entries * (x + 1)
            elif what == "scales":
                ok = passes(scales(x), x // epi_ready)
            else:
                ok = passes(nth(pv, first[x + 1] - 1, 4), (first[x + 1] - 1) >> 2)
            if ok:
                go(ep=ep + 1)
        if not nxt and (pv < nb or ep < len(epi)) and "overwrite" not in faults:
            faults.add("stuck")
        stack += nxt
    return faults


# short items in a row: what one cluster gets when tiles have unions of one or two key blocks
SEQUENCES = [s for n in (2, 3) for s in itertools.product((1, 2), repeat=n)] + \
    [(1, 2, 1, 1), (1, 1, 2, 1), (2, 1, 1, 1), (1, 1, 1, 1), (1, 3, 1, 1), (4, 1, 1), (5, 1, 2)]


@pytest.mark.parametrize("source", ["mla_bf16.cuh", "attn_fp8.cu"])
def test_no_copy_overwrites_a_slot_in_use(source):
    ring = _constants(source)
    bad = [s for s in SEQUENCES if "overwrite" in _explore(s, **ring)]
    assert not bad, bad


@pytest.mark.parametrize("source", ["mla_bf16.cuh", "attn_fp8.cu"])
def test_every_order_of_steps_ends(source):
    # a barrier that completes twice before a waiter looks leaves that waiter behind for good
    ring = _constants(source)
    bad = [s for s in SEQUENCES if _explore(s, **ring)]
    assert not bad, bad
