"""The barrier protocols of the gathering attention kernels (attn_fp8_r64.cuh, attn_fp8.cu, mla_bf16.cuh), run on the CPU.

A CTA, or a pair, is a set of agents -- gather warps, copies in flight, QK^T and PV issue, MMAs in flight, softmax
groups, validity bits, epilogue --, each a list of steps.  Their waits test mbarriers by parity, which answers for the right
phase only while a waiter is at most one phase behind and every arrival falls into the phase it is meant for: every wait
and every arrival is checked against the phase it means.  What the barriers protect -- ring slots, S buffers, O, P, Q's
place, exchanged maxima and sums -- has an owner and a generation: a write that begins while the generation before is
still being written or read is a fault, and so is a read of another generation than the one meant.

The steps are taken in random orders with changing priorities (an agent can be held up for as long as any other can go
on), and for short items in every order.  That the models follow the kernels is checked in two ways: the barriers that
each role waits for are read from the sources, and without any one of its waits, but for those listed as implied by others, a
model has a fault."""
import itertools
import random
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "litetopk_b200" / "csrc"
SRC = {f: re.sub(r"//(?! -{20})[^\n]*", "", (CSRC / f).read_text()) for f in ("attn_fp8_r64.cuh", "attn_fp8.cu", "mla_bf16.cuh")}


def _const(name, src):
    return int(re.search(r"\b%s = (\d+)" % name, SRC[src]).group(1))


class Model:
    """Steps: (kind, what, number).  wait / arrive: barrier, phase; issue: the n-th asynchronous operation of another
    agent may end from here on; after: ... and does; wb / we, rb / re: begin and end of a write, a read of a generation."""

    def __init__(self, inline=False):
        self.steps, self.inline = {}, inline

    def do(self, agent, kind, what, n=0):
        self.steps.setdefault(agent, []).append((kind, what, n))

    def wait(self, agent, bar, phase):
        self.do(agent, "wait", bar, phase)

    def ar(self, agent, bar, phase):
        self.do(agent, "arrive", bar, phase)

    def use(self, agent, *what):            # ("r" | "w", resource, generation) ...: all begun, then all ended
        for kind, res, gen in what:
            self.do(agent, kind + "b", res, gen)
        for kind, res, gen in what:
            self.do(agent, kind + "e", res, gen)

    def later(self, agent, other, uses, arrivals):      # an operation that ends some time later, in order, and arrives then
        for kind, res, gen in uses:
            self.do(agent, kind + "b", res, gen)
        end = agent if self.inline else other
        if not self.inline:
            self.do(agent, "issue", other)
            self.do(other, "after", other)
        for kind, res, gen in uses:
            self.do(end, kind + "e", res, gen)
        for bar, phase in arrivals:
            self.ar(end, bar, phase)

    def roles(self):
        """role -> barriers it waits for (names without their numbers)"""
        out = {}
        for agent, steps in self.steps.items():
            for kind, what, _ in steps:
                if kind == "wait" and not what.startswith("bar_"):      # (bar.sync of a group of warps)
                    out.setdefault(agent.split(".")[0], set()).add(what.split(".")[0])
        return out


def rows64(blocks, bf16_q=False, moves=lambda kb, w: False, warps=(0, 1), inline=False):
    """attn_fp8_r64.cuh: one CTA; two warps per gather set (0 requests Q).  `warps`: of a softmax group (0 publishes)."""
    f = "attn_fp8_r64.cuh"
    slots, groups = _const("kSlots", f), _const("kGroups", f)
    assert re.search(r"uint64_t k_land\[8\], qk_done\[8\], p_ready\[8\], pv_done\[8\];", SRC[f])
    m = Model(inline)
    e = kb0 = o_gen = 0
    q_entry, o_last = [], []
    for it, nb in enumerate([*blocks, 0]):          # behind the last item: an entry to stage its output in
        q_entry.append(e)
        for s, w in itertools.product((0, 1), (0, 1)):
            g, land = f"gather.{s}{w}", f"land.{s}{w}"
            asks = e % 2 == s and w == 0
            if it > 0:
                m.wait(g, "q_taken", it - 1)
            if bf16_q and nb:
                m.wait(g, "q_codes", it)
            if e % 2 == s and e >= slots:
                m.wait(g, f"slot_free.{e % slots}", e // slots - 1)
            if not asks or nb == 0:
                m.ar(g, "q_land", it)
            else:
                m.later(g, "q_copy", [("w", f"lat.{e % slots}", 2 * e), ("w", f"rope.{e % slots}", 2 * e)] +
                        ([("r", f"codes.{it & 1}", it)] if bf16_q else []), [("q_land", it)])
            for k in range(nb):
                x, kb = e + 1 + k, kb0 + k
                if x % 2 == s:
                    if x >= slots:
                        m.wait(g, f"slot_free.{x % slots}", x // slots - 1)
                    m.later(g, land, [("w", f"lat.{x % slots}", 2 * x), ("w", f"rope.{x % slots}", 2 * x)], [(f"k_land.{kb & 7}", kb >> 3)])
        for k in range(nb):
            kb, x = kb0 + k, e + 1 + k
            g, before, behind = kb % groups, (kb - 1) % groups, (kb + 1) % groups
            lat, rope = f"lat.{x % slots}", f"rope.{x % slots}"
            move = {w: k == 0 or moves(kb, w) for w in warps}
            if k == 0 or any(move.values()):
                o_gen += 1                               # O: its item's first PV, or brought to another running max ...
            for i in (0, 1):
                if k == 0:
                    m.wait(f"qk.{i}", "qt_ready", it)
                if kb % 2 == i:
                    m.wait(f"qk.{i}", f"k_land.{kb & 7}", kb >> 3)
                    if kb >= groups:
                        m.wait(f"qk.{i}", f"s_free.{g}", kb // groups - 1)
                    m.later(f"qk.{i}", f"qk_mma.{i}", [("r", lat, 2 * x), ("r", rope, 2 * x), ("r", "q", it), ("w", f"s.{g}", kb)],
                            [(f"qk_done.{kb & 7}", kb >> 3)])
                if k == nb - 1:
                    m.later(f"qk.{i}", f"qk_mma.{i}", [], [("q_free", it)])
            for w in warps:
                a = f"softmax.{g}{w}"
                m.wait(a, f"qk_done.{kb & 7}", kb >> 3)
                m.do(a, "rb", f"s.{g}", kb)
                m.wait(a, f"valid_ready.{g}", kb // groups)
                m.use(a, ("r", f"valid.{g}", kb))
                m.use(a, ("w", f"xbuf.{g}", kb))
                m.ar(a, f"bar_group.{g}", kb // groups)
                m.wait(a, f"bar_group.{g}", kb // groups)
                m.use(a, ("r", f"xbuf.{g}", kb))
                m.do(a, "re", f"s.{g}", kb)
                m.ar(a, f"s_free.{g}", kb // groups)
                m.ar(a, f"valid_free.{g}", kb // groups)
                if kb > 0:
                    m.wait(a, f"m_pub.{before}", (kb - 1) // groups)
                if k > 0:
                    m.use(a, ("r", f"mshare.{before}", kb - 1))
                if move[w] and k + 1 < nb:      # the next block's maxima
                    m.wait(a, f"s_free.{behind}", (kb + 1) // groups)
                    m.use(a, ("r", f"xbuf.{behind}", kb + 1))
                if w == 0:
                    m.use(a, ("w", f"mshare.{g}", kb))
                m.ar(a, f"m_pub.{g}", kb // groups)
                m.use(a, ("w", rope, 2 * x + 1))         # P
                if move[w] and k > 0:
                    m.wait(a, f"pv_done.{(kb - 1) & 7}", (kb - 1) >> 3)
                    m.use(a, ("w", "o", o_gen))
                m.ar(a, f"p_ready.{kb & 7}", kb >> 3)
            if k > 0 and any(move.values()):
                o_gen += 1                               # ... and the PVs behind that
            if k == 0 and it > 0:
                m.wait("pv", "o_free", it - 1)
            m.wait("pv", f"p_ready.{kb & 7}", kb >> 3)
            m.later("pv", "pv_mma", [("r", lat, 2 * x), ("r", rope, 2 * x + 1), ("w", "o", o_gen)],
                    [(f"slot_free.{x % slots}", x // slots), (f"pv_done.{kb & 7}", kb >> 3)])
            if kb >= groups:
                m.wait("valid", f"valid_free.{g}", kb // groups - 1)
            m.use("valid", ("w", f"valid.{g}", kb))
            m.ar("valid", f"valid_ready.{g}", kb // groups)
        for g, w in itertools.product(range(groups if nb else 0), warps):
            if it > 0:
                m.wait(f"softmax.{g}{w}", "fin_free", it - 1)
            m.use(f"softmax.{g}{w}", ("w", f"fin.{g}", it))
            m.ar(f"softmax.{g}{w}", "fin_ready", it)
        o_last.append(o_gen)
        e += nb + 1
        kb0 += nb
    last = -1
    for it in range(-1, len(blocks)):
        n = q_entry[it + 1]
        lat, rope = f"lat.{n % slots}", f"rope.{n % slots}"
        if it + 1 < len(blocks):
            if bf16_q:
                m.use("epilogue", ("w", f"codes.{(it + 1) & 1}", it + 1))
                m.ar("epilogue", "q_codes", it + 1)
            if it >= 0:
                m.wait("epilogue", "q_free", it)
            m.wait("epilogue", "q_land", it + 1)
            m.use("epilogue", ("r", lat, 2 * n), ("r", rope, 2 * n), ("w", "q", it + 1))
            m.ar("epilogue", "qt_ready", it + 1)
            m.ar("epilogue", "q_taken", it + 1)
        else:
            m.wait("epilogue", "q_land", it + 1)
        if it >= 0:
            last += blocks[it]
            m.wait("epilogue", "fin_ready", it)
            m.use("epilogue", *(("r", f"fin.{g}", it) for g in range(groups)))
            m.ar("epilogue", "fin_free", it)
            m.wait("epilogue", f"pv_done.{last & 7}", last >> 3)
            m.use("epilogue", ("r", "o", o_last[it]))
            m.ar("epilogue", "o_free", it)
            m.use("epilogue", ("w", lat, 2 * n + 1))     # output staged in the slot, read out before it is released
            m.use("epilogue", ("r", lat, 2 * n + 1))
        m.ar("epilogue", f"slot_free.{n % slots}", n // slots)
    return m


def pair(blocks, bf16_q=False, moves=lambda kb, w: False, warps=(0, 1), inline=False, ctas=(0, 1), v_warps=(0, 1), f="attn_fp8.cu",
         q_entries=1, q_depth=1):
    """attn_fp8.cu and mla_bf16.cuh: the CTAs of a 128-row tile (barriers of the leader alone end in "L"); two warps each for K (0
    requests Q) and V rows.  `warps`: of a softmax group (0 publishes)."""
    slots = _const("kSlots", f)
    for name, n in (("k_peer", 8), ("v_peer", 8), ("qk_done", 8), ("pv_done", 4), ("s_free", 2), ("p_ready", 2), ("epi_ready", 2)):
        assert re.search(r"uint64_t [^;]*\b%s\[%d\]" % (name, n), SRC[f]), name
    full = {"k": "k_land", "v": "v_land"} if f == "attn_fp8.cu" else {"k": "k_full", "v": "v_full"}
    p_in_slot = f == "mla_bf16.cuh"                      # half of P in the block's rope chunk
    qks = ("even", "odd") if re.search(r"int mine = warp == kWarpMma \? 0 : 1;", SRC[f]) else ("all",)       # QK^T warps
    m = Model(inline)
    e = kb0 = 0
    o_gen = dict.fromkeys(ctas, 0)
    q_entry, o_last = [], []
    for it, nb in enumerate(blocks):
        q_entry.append(e)
        for c in ctas:
            def slot(x, gen=0, parts="abr"):             # a: the half that the peer's V rows go into, b: the other, r: rope
                return [(f"{part}.{x % slots}{c}", 2 * x + gen) for part in parts]
            for w in (0, 1):
                g = f"k.{w}{c}"
                if it > 0:
                    m.wait(g, f"q_taken.{(it - 1) % q_depth}{c}", (it - 1) // q_depth)
                for x in range(e, e + q_entries):
                    if x >= slots:
                        m.wait(g, f"slot_free.{x % slots}{c}", x // slots - 1)
                    if w == 0 and not bf16_q:
                        m.later(g, f"q_copy.{c}", [("w", *r) for r in slot(x)], [(f"q_land.{c}", it)])
                if w != 0 or bf16_q:                     # (bf16: the epilogue warps fill the slot)
                    m.ar(g, f"q_land.{c}", it)
                for k in range(nb):
                    x, kb = e + q_entries + k, kb0 + k
                    if x >= slots:
                        m.wait(g, f"slot_free.{x % slots}{c}", x // slots - 1)
                    m.later(g, f"k_copy.{w}{c}", [("w", *r) for r in slot(x)], [(f"{full['k']}.{kb & 7}{c}", kb >> 3)])
                    if w not in v_warps:
                        continue
                    m.wait(f"v.{w}{c}", f"qk_done.{kb & 7}{c}", kb >> 3)
                    m.later(f"v.{w}{c}", f"v_copy.{w}{c}", [("w", *r) for r in slot(x, 1, "a")], [(f"{full['v']}.{kb & 7}{c}", kb >> 3)])
        for k in range(nb):
            kb, x, g = kb0 + k, e + q_entries + k, (kb0 + k) & 1
            if 1 in ctas:
                for what in "kv":                        # the peer's relays
                    m.wait(f"relay.{what}", f"{full[what]}.{kb & 7}1", kb >> 3)
                    m.ar(f"relay.{what}", f"{what}_peer.{kb & 7}L", kb >> 3)
            qk, qk_mma = (f"qk.{qks[kb % len(qks)]}", f"qk_mma.{qks[kb % len(qks)]}")
            if k == 0:
                for i in qks:                            # both warps, whoever's the block is
                    m.wait(f"qk.{i}", "qt_ready.L", it)
                    if p_in_slot:
                        m.wait(f"qk.{i}", "q_res.L", it)
            m.wait(qk, f"{full['k']}.{kb & 7}0", kb >> 3)
            if 1 in ctas:
                m.wait(qk, f"k_peer.{kb & 7}L", kb >> 3)
            if kb >= 2:
                m.wait(qk, f"s_free.{g}L", (kb >> 1) - 1)
            uses = []
            for c in ctas:
                uses += [("r", f"{part}.{x % slots}{c}", 2 * x) for part in "abr"] + [("r", f"q.{c}", it), ("w", f"s.{g}{c}", kb)] + \
                    ([("r", f"q_res.{c}", it)] if p_in_slot else [])
            m.later(qk, qk_mma, uses, [(f"qk_done.{kb & 7}{c}", kb >> 3) for c in ctas])
            if k == nb - 1:
                for i in qks:
                    m.later(f"qk.{i}", f"qk_mma.{i}", [], [(f"q_free.{c}", it) for c in ctas])
            for c in ctas:
                if kb >= 2:
                    m.wait(f"valid.{c}", f"valid_free.{g}{c}", (kb >> 1) - 1)
                m.use(f"valid.{c}", ("w", f"valid_bits.{g}{c}", kb))
                m.ar(f"valid.{c}", f"valid_ready.{g}{c}", kb >> 1)
                move = {w: k > 0 and moves(kb, w + 2 * c) for w in warps}
                if k == 0 or any(move.values()):
                    o_gen[c] += 1
                for w in warps:
                    a = f"softmax.{g}{w}{c}"
                    m.wait(a, f"qk_done.{kb & 7}{c}", kb >> 3)
                    m.use(a, ("r", f"s.{g}{c}", kb))
                    m.ar(a, f"s_free.{g}L", kb >> 1)
                    m.wait(a, f"valid_ready.{g}{c}", kb >> 1)
                    m.use(a, ("r", f"valid_bits.{g}{c}", kb))
                    m.ar(a, f"valid_free.{g}{c}", kb >> 1)
                    m.use(a, ("w", f"xbuf.{kb & 3}{c}", kb))       # [group][parity of the group's block]
                    m.ar(a, f"bar_group.{g}{c}", kb >> 1)
                    m.wait(a, f"bar_group.{g}{c}", kb >> 1)
                    m.use(a, ("r", f"xbuf.{kb & 3}{c}", kb))
                    if k > 0:
                        m.wait(a, f"m_pub.{g ^ 1}{c}", (kb - 1) >> 1)
                        m.use(a, ("r", f"mshare.{g ^ 1}{c}", kb - 1))
                    if w == 0:
                        m.use(a, ("w", f"mshare.{g}{c}", kb))
                    m.ar(a, f"m_pub.{g}{c}", kb >> 1)
                    if kb >= 2:
                        m.wait(a, f"pv_done.{(kb - 2) & 3}{c}", (kb - 2) >> 2)
                    m.use(a, ("w", f"p.{g}{c}", kb), *([("w", f"r.{x % slots}{c}", 2 * x + 1)] if p_in_slot else []))
                    if move[w]:
                        m.wait(a, f"pv_done.{(kb - 1) & 3}{c}", (kb - 1) >> 2)
                        m.use(a, ("w", f"o.{c}", o_gen[c]))
                    m.ar(a, f"p_ready.{g}L", kb >> 1)
                if any(move.values()):
                    o_gen[c] += 1
            m.wait("pv", f"{full['v']}.{kb & 7}0", kb >> 3)
            if 1 in ctas:
                m.wait("pv", f"v_peer.{kb & 7}L", kb >> 3)
            if k == 0 and it > 0:
                m.wait("pv", "o_free.L", it - 1)
            m.wait("pv", f"p_ready.{g}L", kb >> 1)
            uses = []
            for c in ctas:
                uses += [("r", f"a.{x % slots}{c}", 2 * x + 1), ("r", f"b.{x % slots}{c}", 2 * x), ("r", f"p.{g}{c}", kb),
                         ("w", f"o.{c}", o_gen[c])] + ([("r", f"r.{x % slots}{c}", 2 * x + 1)] if p_in_slot else [])
            m.later("pv", "pv_mma", uses, [(f"slot_free.{x % slots}{c}", x // slots) for c in ctas] +
                    [(f"pv_done.{kb & 3}{c}", kb >> 2) for c in ctas])
        for c in ctas:
            for a in (f"softmax.{g}{w}{c}" for g in (0, 1) for w in warps):
                if it > 0:
                    m.wait(a, f"epi_ready.{(it - 1) & 1}{c}", (it - 1) >> 1)
                m.use(a, ("w", f"fin.{c}", it))
                m.ar(a, f"bar_end.{c}", it)
                m.wait(a, f"bar_end.{c}", it)
                if a == f"softmax.00{c}":
                    m.use(a, ("r", f"fin.{c}", it), ("w", f"oscale.{it & 1}{c}", it))
                m.ar(a, f"epi_ready.{it & 1}{c}", it >> 1)
        o_last.append(dict(o_gen))
        e += nb + q_entries
        kb0 += nb
    for c in ctas:
        last, epi = -1, f"epilogue.{c}"
        for it in range(-1, len(blocks)):
            if it + 1 < len(blocks):
                n = q_entry[it + 1]
                entries = [(f"{part}.{x % slots}{c}", 2 * x) for x in range(n, n + q_entries) for part in "abr"]
                if bf16_q:
                    m.wait(epi, f"q_land.{c}", it + 1)
                    m.use(epi, *(("w", *r) for r in entries))
                if it >= 0:
                    m.wait(epi, f"q_free.{c}", it)
                if p_in_slot:                            # the resident chunks
                    m.later(epi, f"q_res_copy.{c}", [("w", f"q_res.{c}", it + 1)], [("q_res.L", it + 1)])
                if not bf16_q:
                    m.wait(epi, f"q_land.{c}", it + 1)
                m.use(epi, *(("r", *r) for r in entries), ("w", f"q.{c}", it + 1))
                m.ar(epi, "qt_ready.L", it + 1)
                for x in range(n, n + q_entries):
                    m.ar(epi, f"slot_free.{x % slots}{c}", x // slots)
                m.ar(epi, f"q_taken.{(it + 1) % q_depth}{c}", (it + 1) // q_depth)
            if it >= 0:
                last += blocks[it]
                m.wait(epi, f"epi_ready.{it & 1}{c}", it >> 1)
                m.wait(epi, f"pv_done.{last & 3}{c}", last >> 2)
                m.use(epi, ("r", f"oscale.{it & 1}{c}", it), ("r", f"o.{c}", o_last[it][c]))
                m.ar(epi, "o_free.L", it)
                if it + 1 == len(blocks):                # the last item's output, staged in the ring
                    m.use(epi, *(("w", f"{part}.{x}{c}", 1 << 20) for x in range(slots) for part in "abr"))
    return m


def bf16(blocks, bf16_q=False, **kw):                    # (its queries are bf16: nothing to quantise)
    return pair(blocks, False, f="mla_bf16.cuh", q_entries=_const("kQEntries", "mla_bf16.cuh"), q_depth=2, **kw)


class Run:
    """The state of a model on its way; step(agent) is False if it has to wait, True if it went on, else what went wrong."""

    def __init__(self, model, without=None):
        names = {k: i for i, k in enumerate(model.steps)}
        bars, res, need = {}, {}, {}
        self.ends = {}                                   # (resource, generation) -> writes and reads that it has
        self.steps = []
        for agent, steps in model.steps.items():
            out = []
            for kind, what, n in steps:
                if kind in ("wait", "arrive"):
                    if kind == "wait" and (agent.split(".")[0], what.split(".")[0]) == without:
                        continue
                    i = bars.setdefault(what, len(bars))
                    if kind == "arrive":
                        need.setdefault(i, {}).setdefault(n, 0)
                        need[i][n] += 1
                elif kind in ("issue", "after"):
                    i = names[what]
                else:
                    i = res.setdefault(what, len(res))
                    if kind[1] == "e":
                        self.ends.setdefault((i, n), [0, 0])[kind == "re"] += 1
                out.append((kind, i, n))
            self.steps.append(out)
        for phases in need.values():
            assert len(set(phases.values())) == 1 and sorted(phases) == list(range(len(phases)))
        self.names, self.bars, self.res = list(names), list(bars), list(res)
        self.need = [next(iter(need[i].values())) for i in range(len(bars))]
        self.pos, self.issued, self.done = ([0] * len(names) for _ in range(3))
        self.completed, self.pending = [0] * len(bars), [0] * len(bars)
        self.gen, self.count = [None] * len(res), [[0, 0] for _ in res]     # the present generation; its writes, reads ended

    def passes(self, bar, phase):
        return (self.completed[bar] & 1) != (phase & 1)

    def step(self, a):
        kind, i, n = self.steps[a][self.pos[a]]
        if kind == "wait":
            if self.completed[i] > n + 1:
                return f"{self.names[a]} waits for phase {n} of {self.bars[i]}, {self.completed[i]} are complete"
            if not self.passes(i, n):
                return False
            if self.completed[i] != n + 1:
                return f"{self.names[a]} passes {self.bars[i]} in phase {self.completed[i]}, {n} was meant"
        elif kind == "arrive":
            if self.completed[i] != n:
                return f"{self.names[a]} arrives on {self.bars[i]} in phase {self.completed[i]}, {n} was meant"
            self.pending[i] += 1
            if self.pending[i] == self.need[i]:
                self.pending[i], self.completed[i] = 0, self.completed[i] + 1
        elif kind == "after":
            if self.done[i] == self.issued[i]:
                return False
            self.done[i] += 1
        elif kind == "issue":
            self.issued[i] += 1
        elif kind == "wb":
            if self.gen[i] != n:
                if self.gen[i] is not None and self.count[i] != self.ends[i, self.gen[i]]:
                    return f"{self.names[a]} overwrites {self.res[i]}, in use"
                self.gen[i], self.count[i] = n, [0, 0]
        elif kind == "rb":
            if self.gen[i] != n or self.count[i][0] != self.ends[i, n][0]:
                return f"{self.names[a]} reads {self.res[i]}, generation {self.gen[i]} for {n}"
        else:
            if self.gen[i] != n:
                return f"{self.names[a]} has lost {self.res[i]}"
            self.count[i] = [self.count[i][0] + (kind == "we"), self.count[i][1] + (kind == "re")]
        self.pos[a] += 1
        return True

    def left(self):
        return [a for a, p in enumerate(self.pos) if p < len(self.steps[a])]

    def where(self):
        return {self.names[a]: self.steps[a][self.pos[a]] for a in self.left()}


def _random_order(run, rng):
    """What went wrong in one random order, or None."""
    order = list(range(len(run.pos)))
    rng.shuffle(order)
    alive = set(run.left())
    while alive:
        if rng.random() < 0.1:
            a = order.pop(rng.randrange(len(order)))
            order.insert(rng.randrange(len(order) + 1), a)
        for a in order:
            if a in alive:
                got = run.step(a)
                if got is True:
                    if run.pos[a] == len(run.steps[a]):
                        alive.discard(a)
                    break
                if got:
                    return got
        else:
            return f"stuck: {run.where()}"
    return None


def _blocks(rng):
    most = rng.choice([1, 2, 3, 9])
    return [rng.randint(1, most) for _ in range(rng.randint(3, 9))]


def _moves(rng):
    p, seed = rng.choice([0.0, 0.2, 1.0]), rng.randrange(1 << 30)
    return lambda kb, w: random.Random(seed + 97 * kb + w).random() < p


KERNELS = [rows64, pair, bf16]
SOURCE = {rows64: "attn_fp8_r64.cuh", pair: "attn_fp8.cu", bf16: "mla_bf16.cuh"}


@pytest.mark.parametrize("bf16_q", [False, True])
@pytest.mark.parametrize("kernel", KERNELS)
def test_no_order_of_the_warps_breaks_the_protocol(kernel, bf16_q):
    rng = random.Random(64 + bf16_q)
    for _ in range(60):
        blocks = _blocks(rng)
        fault = _random_order(Run(kernel(blocks, bf16_q=bf16_q, moves=_moves(rng))), rng)
        assert fault is None, (blocks, fault)


@pytest.mark.parametrize("kernel", KERNELS)
def test_a_model_without_one_of_its_waits_has_a_fault(kernel):
    waits = {(role, bar) for bf16_q in (False, True)
             for role, bars in kernel([3, 1, 2, 9, 2, 1, 1], bf16_q=bf16_q, moves=lambda kb, w: True).roles().items() for bar in bars}
    for without in sorted(waits):          # (within 8 of these runs each)
        rng = random.Random(5)
        assert any(_random_order(Run(kernel(_blocks(rng), bf16_q=bool(i & 1), moves=_moves(rng)), without), rng)
                   for i in range(100)), without


ROLES = {"softmax": "softmax", "KV row gather": "gather", "QK^T issue": "qk", "MMA issue": "qk", "PV issue": "pv", '"landed" relays': "relay",
         "index-validity bits": "valid", "Q in, epilogue": "epilogue", "epilogue warps": "epilogue", "TMA producers": None}


def _roles_of_source(f):
    """role -> its part of the kernel"""
    parts = re.split(r"// -{20,} ([^\n]*)", SRC[f][SRC[f].index("extern __shared__"):])[1:]
    out = {}
    for title, body in zip(parts[::2], parts[1::2]):
        role = next(r for t, r in ROLES.items() if title.startswith(t))
        if role:
            out[role] = out.get(role, "") + body
    return out


@pytest.mark.parametrize("kernel", KERNELS)
def test_the_models_wait_where_the_kernels_wait(kernel):
    want = {}
    for bf16_q in (False, True):
        for role, bars in kernel([3, 1, 2, 9, 2, 1, 1], bf16_q=bf16_q, moves=lambda kb, w: True).roles().items():
            want.setdefault("gather" if role in "kv" else role, set()).update(bars)
    got = {}
    for role, body in _roles_of_source(SOURCE[kernel]).items():
        tested = re.findall(r"mbar_(?:wait|try_wait|test)\(([^,]*),|uint64_t\* bar = ([^;]*);", body)
        got[role] = {bar for args in tested for x in args for bar in re.findall(r"&ms\.(\w+)", x)}
    assert got == want


def _every_order(kernel, blocks, **kw):
    """What goes wrong in any order of the agents' steps; the steps behind a wait go with it, as do asynchronous ends."""
    run = Run(kernel(blocks, inline=True, **kw))
    agents = range(len(run.pos))
    seen, stack = {tuple(run.pos)}, [(run.pos, run.completed, run.pending, run.gen, run.count)]
    while stack:
        state = stack.pop()
        moved = ended = 0
        for a in agents:
            j = state[0][a]
            if j == len(run.steps[a]):
                ended += 1
                continue
            kind, i, n = run.steps[a][j]
            if kind == "wait" and state[1][i] <= n + 1 and (state[1][i] & 1) == (n & 1):
                continue                                 # it has to wait
            run.pos, run.completed, run.pending, run.gen, run.count = (list(x) for x in state)
            got = run.step(a)
            while got is True and run.pos[a] < len(run.steps[a]) and run.steps[a][run.pos[a]][0] != "wait":
                got = run.step(a)
            if got is not True:
                return got
            moved += 1
            key = tuple(run.pos)
            if key not in seen:
                seen.add(key)
                stack.append((run.pos, run.completed, run.pending, run.gen, run.count))
        if not moved and ended < len(agents):
            return "stuck"
    return None


# short items in a row: what a CTA gets when tiles have unions of one or two key blocks (one warp of each softmax group,
# one V warp, and of a pair the leader: all orders of everything are too many)
SHORT = [(1, 1), (1, 2), (2, 1), (1, 1, 1), (1, 2, 1)]


@pytest.mark.parametrize("kernel,sequences,kw", [
    (rows64, SHORT, dict(warps=(0,))),
    (pair, SHORT + [(1, 2, 1, 1), (2, 1, 1, 1)], dict(warps=(0,), ctas=(0,), v_warps=(0,))),
    (bf16, SHORT + [(1, 2, 1, 1), (2, 1, 1, 1)], dict(warps=(0,), ctas=(0,), v_warps=(0,)))])
def test_every_order_of_short_items(kernel, sequences, kw):
    bad = [(s, fault) for s in sequences for fault in [_every_order(kernel, s, **kw)] if fault]
    assert not bad, bad


def _give_up(model, rng, q_entries, leaves, asks_if_all_well):
    """A run in which one arrival never comes, or Q never lands, and once nobody can go on every wait that does not pass gives up.
    Gather and MMA warps leave then (`leaves`; the others fall through), and Q is requested, or a gather warp's arrival
    for it made, only as long as no wait of the CTA has given up (`asks_if_all_well`).  Returns what is wrong with the
    copies in flight, or None."""
    run = Run(model)
    paired = "gather.00" not in run.names                # (QK^T and PV are the leader's, the relays the peer's)
    cta = ["" if not paired else "1" if name.startswith("relay") or name.endswith("1") else "0" for name in run.names]
    role = [name.split(".")[0] for name in run.names]
    arrivals = [(a, j) for a, steps in enumerate(run.steps) for j, (kind, i, _) in enumerate(steps)
                if kind == "arrive" and not run.bars[i].startswith("bar_")]
    lost = rng.choice(arrivals + [None])
    late = rng.choice([0, 1, 2, 1 << 30]) * q_entries    # this and later Qs land when all warps are done
    giving_up, left, gone, gave = False, set(), set(), set()          # (giving up: the limit has run out)
    withheld = set()                                     # arrivals for Q that were passed by

    def step(a):
        kind, i, n = run.steps[a][run.pos[a]]
        bar = run.bars[i].split(".")[0] if kind in ("wait", "arrive") else ""
        if kind == "wait" and not run.passes(i, n):
            if not giving_up or bar.startswith("bar_"):  # (bar.sync does not give up)
                return False
            gave.add(a)
            left.add(cta[a])
            if leaves and role[a] in ("gather", "k", "v", "qk", "pv"):
                gone.add(a)
                return True
        elif kind == "arrive":
            held = bar == "q_land" and not role[a].endswith("copy") and asks_if_all_well and (cta[a] in left or a in gave)
            if held:
                withheld.add((a, run.pos[a]))
            if (a, run.pos[a]) != lost and not held:
                run.pending[i] += 1
                if bar == "q_land" and run.pending[i] > run.need[i]:
                    return f"{run.names[a]} arrives on q_land once more than it counts"
                if run.pending[i] >= run.need[i]:
                    run.pending[i], run.completed[i] = 0, run.completed[i] + 1
        elif kind == "issue":
            if role[i] in ("q_copy", "q_res_copy") and asks_if_all_well and cta[a] in left:
                pass
            elif role[i] in ("land", "q_copy", "k_copy", "v_copy") and a in gave:
                return f"{run.names[a]} requests a copy behind a wait that gave up"
            elif role[i] == "q_copy" and run.issued[i] % q_entries == 0 and run.issued[i] != run.done[i]:
                return f"{run.names[a]} requests Q with another in flight"
            else:
                run.issued[i] += 1
        elif kind == "after":
            if run.done[i] == run.issued[i] or (role[a] == "q_copy" and run.done[i] >= late):
                return False
            run.done[i] += 1
        run.pos[a] += 1
        return True

    order = list(range(len(role)))
    while True:
        if rng.random() < 0.1:
            rng.shuffle(order)
        for a in order:
            if a not in gone and run.pos[a] < len(run.steps[a]):
                got = step(a)
                if got is True:
                    break
                if got:
                    return got
        else:
            if giving_up:
                break
            giving_up = True
    late = 1 << 30
    for i, name in enumerate(run.names):                 # the tear-down
        if role[i] != "q_copy" or run.issued[i] == run.done[i]:
            continue
        if cta[i] not in left:
            return "a block retires with its Q on the way"
        land = run.bars.index("q_land" + ("." + cta[i] if cta[i] else ""))
        items = (run.issued[i] + q_entries - 1) // q_entries
        # the arrivals that are missing for the last Q requested: other gather warps', the second half's
        for a, r in enumerate(role):
            if r in ("gather", "k") and cta[a] == cta[i]:
                made = [j for j, x in enumerate(run.steps[a]) if x[:2] == ("arrive", land) and x[2] == items - 1]
                run.pending[land] += sum(j >= run.pos[a] or (a, j) == lost or (a, j) in withheld for j in made)
        run.pending[land] += items * q_entries - run.issued[i]
        if run.passes(land, items - 1):
            return "the tear-down does not wait for Q"
        run.pending[land] += run.issued[i] - run.done[i]
        if lost is None or lost[0] != i:
            if run.pending[land] != run.need[land]:
                return f"the tear-down counts {run.pending[land]} arrivals of {run.need[land]}"
    return None


@pytest.mark.parametrize("bf16_q", [False, True])
@pytest.mark.parametrize("kernel", KERNELS)
def test_a_launch_that_gives_up_has_no_copy_in_flight_when_it_ends(kernel, bf16_q):
    # the warps' behaviour behind a wait that gave up, read from the source
    src, roles = SRC[SOURCE[kernel]], _roles_of_source(SOURCE[kernel])
    leaves = not re.search(r"(?:[;{}]|if \([^;{}]*?\))\s*mbar_wait\(", roles["gather"]) and "go = __all_sync(0xffffffffu, ok);" in roles["gather"]
    asks = len(re.findall(r"lane == 0 && ok && !wt\.aborting\(\)", roles["gather"])) == 1 and \
        (kernel is not bf16 or bool(re.search(r"auto request_q = [^;]*;\s*if \(wt\.aborting\(\)\) return;", src)))
    end = src[src.index("if (ms.left != 0) {"):]
    assert all(x in end for x in ("cp_async_wait_all();", "mbar_drain(&ms.q_land,", "mbar_drain(&ms.qk_done[", "mbar_drain(&ms.pv_done["))
    entries = _const("kQEntries", SOURCE[kernel]) if kernel is bf16 else 1

    def faults(leaves, asks):
        rng = random.Random(9)
        return {f for _ in range(200) for f in [_give_up(kernel(_blocks(rng), bf16_q=bf16_q, moves=_moves(rng)), rng, entries,
                                                         leaves, asks)] if f}
    assert not faults(leaves, asks)
    assert any("behind a wait" in f for f in faults(False, asks))
    if kernel is rows64 or not bf16_q:                   # (of a pair's bf16 queries nothing is requested from TMA)
        assert any("another in flight" in f or "once more" in f for f in faults(True, False))
