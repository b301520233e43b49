"""The barrier protocols of the gathering attention kernels (attn_fp8_r64.cuh, attn_fp8.cu, mla_bf16.cuh), run on the CPU
in random orders.

Their warps wait on mbarriers by parity, which answers for the right phase only while a waiter is at most
one phase behind and every arrival falls into the phase it is meant for.  A CTA, or a pair, is a set of agents --
gather sets, copies in flight, QK^T and PV issue, MMAs in flight, softmax groups, validity bits, epilogue --
whose steps are taken in orders with random and changing priorities (an agent can be held up for
as long as any other can go on); every wait and every arrival is checked against the phase it means."""
import random
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "litetopk_b200" / "csrc"
SRC, SRC_PAIR, SRC_BF16 = ((CSRC / f).read_text() for f in ("attn_fp8_r64.cuh", "attn_fp8.cu", "mla_bf16.cuh"))


def _const(name, src=SRC):
    return int(re.search(r"\b%s = (\d+)" % name, src).group(1))


def _agents(blocks, bf16_q, rescale):
    """name -> steps ("wait" | "arrive" | "issue" | "after", barrier or agent, phase or count); barrier -> arrivals"""
    slots, groups = _const("kSlots"), _const("kGroups")
    assert re.search(r"uint64_t k_land\[8\], qk_done\[8\], p_ready\[8\], pv_done\[8\];", SRC)
    a = {k: [] for k in ("g00", "g01", "g10", "g11", "land00", "land01", "land10", "land11", "qland00", "qland01", "qland10",
                         "qland11", "qk0", "qk1", "qkp0", "qkp1", "pv", "pvp", "valid", "epi",
                         *(f"s{g}{w}" for g in range(groups) for w in (0, 1)))}
    need = {}

    def ar(agent, bar, phase, n=1):
        need[bar] = n
        a[agent].append(("arrive", bar, phase))

    def issue(agent, other):      # the n-th asynchronous operation of `other` may complete from here on
        a[agent].append(("issue", other, 0))

    def after(agent):             # ... and does
        a[agent].append(("after", agent, 0))

    def wait(agent, bar, phase):
        a[agent].append(("wait", bar, phase))

    e = kb0 = 0
    q_entry = []
    for it, nb in enumerate([*blocks, 0]):          # behind the last item: an entry to stage its output in
        q_entry.append(e)
        for s in (0, 1):
            for w in (0, 1):
                g, land = f"g{s}{w}", f"land{s}{w}"
                if it > 0:
                    wait(g, "q_taken", it - 1)
                if bf16_q and nb:
                    wait(g, "q_codes", it)
                if e % 2 == s:
                    if e >= slots:
                        wait(g, f"slot_free{e % slots}", e // slots - 1)
                issue(g, f"qland{s}{w}")
                after(f"qland{s}{w}")
                ar(f"qland{s}{w}", "q_land", it, 4)
                for k in range(nb):
                    x, kb = e + 1 + k, kb0 + k
                    if x % 2 == s:
                        if x >= slots:
                            wait(g, f"slot_free{x % slots}", x // slots - 1)
                        issue(g, land)
                        after(land)
                        ar(land, f"k_land{kb & 7}", kb >> 3, 2)
        for k in range(nb):
            kb, x = kb0 + k, e + 1 + k
            for m in (0, 1):
                if k == 0:
                    wait(f"qk{m}", "qt_ready", it)
                if kb % 2 == m:
                    wait(f"qk{m}", f"k_land{kb & 7}", kb >> 3)
                    if kb >= groups:
                        wait(f"qk{m}", f"s_free{kb % groups}", kb // groups - 1)
                    issue(f"qk{m}", f"qkp{m}")
                    after(f"qkp{m}")
                    ar(f"qkp{m}", f"qk_done{kb & 7}", kb >> 3)
                if k == nb - 1:
                    issue(f"qk{m}", f"qkp{m}")
                    after(f"qkp{m}")
                    ar(f"qkp{m}", "q_free", it, 2)
            if k == 0 and it > 0:
                wait("pv", "o_free", it - 1)
            wait("pv", f"p_ready{kb & 7}", kb >> 3)
            issue("pv", "pvp")
            after("pvp")
            ar("pvp", f"slot_free{x % slots}", x // slots)
            ar("pvp", f"pv_done{kb & 7}", kb >> 3)
            if kb >= groups:
                wait("valid", f"valid_free{kb % groups}", kb // groups - 1)
            ar("valid", f"valid_ready{kb % groups}", kb // groups)
            g, before = kb % groups, (kb - 1) % groups
            for w in (0, 1):
                s = f"s{g}{w}"
                wait(s, f"qk_done{kb & 7}", kb >> 3)
                wait(s, f"valid_ready{g}", kb // groups)
                ar(s, f"group{g}", kb // groups, 2)
                wait(s, f"group{g}", kb // groups)
                ar(s, f"s_free{g}", kb // groups, 2)
                ar(s, f"valid_free{g}", kb // groups, 2)
                if kb > 0:
                    wait(s, f"m_pub{before}", (kb - 1) // groups)
                if (rescale or k == 0) and k + 1 < nb:      # the next block's maxima
                    wait(s, f"s_free{(g + 1) % groups}", (kb + 1) // groups)
                ar(s, f"m_pub{g}", kb // groups, 2)
                if rescale and k > 0:
                    wait(s, f"pv_done{(kb - 1) & 7}", (kb - 1) >> 3)
                ar(s, f"p_ready{kb & 7}", kb >> 3, 2)
        for g in range(groups if nb else 0):
            for w in (0, 1):
                if it > 0:
                    wait(f"s{g}{w}", "fin_free", it - 1)
                ar(f"s{g}{w}", "fin_ready", it, 2 * groups)
        e += nb + 1
        kb0 += nb
    last = -1
    for it in range(-1, len(blocks)):
        staged = f"slot_free{q_entry[it + 1] % slots}"
        if it + 1 < len(blocks):
            if bf16_q:
                ar("epi", "q_codes", it + 1)
            if it >= 0:
                wait("epi", "q_free", it)
            wait("epi", "q_land", it + 1)
            ar("epi", "qt_ready", it + 1)
            ar("epi", "q_taken", it + 1)
        else:
            wait("epi", "q_land", it + 1)
        if it >= 0:
            last += blocks[it]
            wait("epi", "fin_ready", it)
            ar("epi", "fin_free", it)
            wait("epi", f"pv_done{last & 7}", last >> 3)
            ar("epi", "o_free", it)
        ar("epi", staged, q_entry[it + 1] // slots)
    return a, need


def _pair_agents(blocks, bf16_q, rescale, src=SRC_PAIR, q_entries=1, q_depth=1):
    """The same for the two CTAs that share a 128-row tile; names and barriers end in their CTA ("L": the leader's)."""
    slots = _const("kSlots", src)
    for name, n in (("k_peer", 8), ("v_peer", 8), ("qk_done", 8), ("pv_done", 4), ("s_free", 2), ("p_ready", 2), ("epi_ready", 2)):
        assert re.search(r"uint64_t [^;]*\b%s\[%d\]" % (name, n), src), name
    a, need = {}, {}

    def do(agent, kind, what, phase=0):
        a.setdefault(agent, []).append((kind, what, phase))

    def ar(agent, bar, phase, n=1):
        need[bar] = n
        do(agent, "arrive", bar, phase)

    def async_ar(agent, other, bar, phase, n=1):       # started by `agent`, arrives some time later, in order
        do(agent, "issue", other)
        do(other, "after", other)
        ar(other, bar, phase, n)

    def wait(agent, bar, phase):
        do(agent, "wait", bar, phase)

    e = kb0 = 0
    q_entry = []
    for it, nb in enumerate(blocks):
        q_entry.append(e)
        for c in (0, 1):
            for w in (0, 1):
                g = f"k{w}{c}"
                if it > 0:
                    wait(g, f"q_taken{(it - 1) % q_depth}{c}", (it - 1) // q_depth)
                for x in range(e, e + q_entries):
                    if x >= slots:
                        wait(g, f"slot_free{x % slots}{c}", x // slots - 1)
                    if w == 0:
                        async_ar(g, f"qland{w}{c}", f"q_land{c}", it, q_entries + 1)
                if w == 1:
                    async_ar(g, f"qland{w}{c}", f"q_land{c}", it, q_entries + 1)
                for k in range(nb):
                    x, kb = e + q_entries + k, kb0 + k
                    if x >= slots:
                        wait(g, f"slot_free{x % slots}{c}", x // slots - 1)
                    async_ar(g, f"kland{w}{c}", f"k_land{kb & 7}{c}", kb >> 3, 2)
                    wait(f"v{w}{c}", f"qk_done{kb & 7}{c}", kb >> 3)
                    async_ar(f"v{w}{c}", f"vland{w}{c}", f"v_land{kb & 7}{c}", kb >> 3, 2)
        for k in range(nb):
            kb, x = kb0 + k, e + q_entries + k
            for what in "kv":                         # the peer's relays
                wait(f"r{what}", f"{what}_land{kb & 7}1", kb >> 3)
                ar(f"r{what}", f"{what}_peer{kb & 7}L", kb >> 3)
            if k == 0:
                wait("qk", "qt_readyL", it)
            wait("qk", f"k_land{kb & 7}0", kb >> 3)
            wait("qk", f"k_peer{kb & 7}L", kb >> 3)
            if kb >= 2:
                wait("qk", f"s_free{kb & 1}L", (kb >> 1) - 1)
            for c in (0, 1):
                async_ar("qk", "qkp", f"qk_done{kb & 7}{c}", kb >> 3)
            if k == nb - 1:
                for c in (0, 1):
                    async_ar("qk", "qkp", f"q_free{c}", it)
            wait("pv", f"v_land{kb & 7}0", kb >> 3)
            wait("pv", f"v_peer{kb & 7}L", kb >> 3)
            if k == 0 and it > 0:
                wait("pv", "o_freeL", it - 1)
            wait("pv", f"p_ready{kb & 1}L", kb >> 1)
            for c in (0, 1):
                async_ar("pv", "pvp", f"slot_free{x % slots}{c}", x // slots)
                async_ar("pv", "pvp", f"pv_done{kb & 3}{c}", kb >> 2)
            g = kb & 1
            for c in (0, 1):
                if kb >= 2:
                    wait(f"valid{c}", f"valid_free{g}{c}", (kb >> 1) - 1)
                ar(f"valid{c}", f"valid_ready{g}{c}", kb >> 1)
                for w in (0, 1):
                    s = f"s{g}{w}{c}"
                    wait(s, f"qk_done{kb & 7}{c}", kb >> 3)
                    ar(s, f"s_free{g}L", kb >> 1, 4)
                    wait(s, f"valid_ready{g}{c}", kb >> 1)
                    ar(s, f"valid_free{g}{c}", kb >> 1, 2)
                    ar(s, f"group{g}{c}", kb >> 1, 2)
                    wait(s, f"group{g}{c}", kb >> 1)
                    if k > 0:
                        wait(s, f"m_pub{g ^ 1}{c}", (kb - 1) >> 1)
                    ar(s, f"m_pub{g}{c}", kb >> 1, 2)
                    if kb >= 2:
                        wait(s, f"pv_done{(kb - 2) & 3}{c}", (kb - 2) >> 2)
                    if rescale and k > 0:
                        wait(s, f"pv_done{(kb - 1) & 3}{c}", (kb - 1) >> 2)
                    ar(s, f"p_ready{g}L", kb >> 1, 4)
        for c in (0, 1):
            for s in (f"s{g}{w}{c}" for g in (0, 1) for w in (0, 1)):
                if it > 0:
                    wait(s, f"epi_ready{(it - 1) & 1}{c}", (it - 1) >> 1)
                ar(s, f"end{c}", it, 4)
                wait(s, f"end{c}", it)
                ar(s, f"epi_ready{it & 1}{c}", it >> 1, 4)
        e += nb + q_entries
        kb0 += nb
    for c in (0, 1):
        last, epi = -1, f"epi{c}"
        for it in range(-1, len(blocks)):
            if it + 1 < len(blocks):
                order = [(f"q_land{c}", it + 1), (f"q_free{c}", it)]
                for bar, phase in order if bf16_q else order[::-1]:
                    if phase >= 0:
                        wait(epi, bar, phase)
                ar(epi, "qt_readyL", it + 1, 2)
                for x in range(q_entry[it + 1], q_entry[it + 1] + q_entries):
                    ar(epi, f"slot_free{x % slots}{c}", x // slots)
                ar(epi, f"q_taken{(it + 1) % q_depth}{c}", (it + 1) // q_depth)
            if it >= 0:
                last += blocks[it]
                wait(epi, f"epi_ready{it & 1}{c}", it >> 1)
                wait(epi, f"pv_done{last & 3}{c}", last >> 2)
                ar(epi, "o_freeL", it, 2)
    return a, need


def _bf16_agents(blocks, bf16_q, rescale):
    return _pair_agents(blocks, bf16_q, rescale, SRC_BF16, _const("kQEntries", SRC_BF16), 2)


def _run(agents, need, rng):
    """One random order; returns what went wrong, or None."""
    pos, issued, done = dict.fromkeys(agents, 0), dict.fromkeys(agents, 0), dict.fromkeys(agents, 0)
    completed, pending = dict.fromkeys(need, 0), dict.fromkeys(need, 0)
    prio = {k: rng.random() for k in agents}
    while True:
        if rng.random() < 0.1:
            prio[rng.choice(list(prio))] = rng.random()
        for name in sorted(agents, key=prio.get):
            steps = agents[name]
            if pos[name] == len(steps):
                continue
            kind, what, phase = steps[pos[name]]
            if kind == "wait":
                if completed[what] > phase + 1:
                    return f"{name} waits for phase {phase} of {what}, {completed[what]} are complete"
                if (completed[what] & 1) == (phase & 1):
                    continue
                if completed[what] != phase + 1:
                    return f"{name} passes {what} in phase {completed[what]}, {phase} was meant"
            elif kind == "after":
                if done[name] == issued[name]:
                    continue
                done[name] += 1
            elif kind == "issue":
                issued[what] += 1
            else:
                if completed[what] != phase:
                    return f"{name} arrives on {what} in phase {completed[what]}, {phase} was meant"
                pending[what] += 1
                if pending[what] == need[what]:
                    pending[what], completed[what] = 0, completed[what] + 1
            pos[name] += 1
            break
        else:
            stuck = {k: agents[k][p] for k, p in pos.items() if p < len(agents[k])}
            return f"stuck: {stuck}" if stuck else None


@pytest.mark.parametrize("bf16_q", [False, True])
@pytest.mark.parametrize("rescale", [False, True])
@pytest.mark.parametrize("agents", [_agents, _pair_agents, _bf16_agents])
def test_no_order_of_the_warps_breaks_a_phase(agents, bf16_q, rescale):
    rng = random.Random(64 + 2 * bf16_q + rescale)
    for n in range(100):
        most = rng.choice([1, 2, 3, 9])
        blocks = [rng.randint(1, most) for _ in range(rng.randint(3, 9))]
        fault = _run(*agents(blocks, bf16_q, rescale), rng)
        assert fault is None, (blocks, fault)
