"""Hand-over between the softmax groups, the PV issuer and the epilogue of the forward strip kernel, checked on the planner's own
block streams without a GPU.

A wait on a barrier knows its phase by parity only: with k completions to wait for it passes at k, and also at k - 2, but not at k + 1.
It is right if k - 1 of them are certain when it starts, and the one after the k'th cannot come before it has passed, whatever the
roles' speed.  What is certain is worked out here with vector clocks: every event knows the latest event of every role that
must have come before it (program order, and the waits)."""
import ctypes as C
import random
import re

import pytest
import torch

from test_gpu_strip_roles import STREAMS
from test_kernel_sources import source

from dl_templates_b200 import _lib


def rules():
    """How the kernel's source takes the parity of its waits for O_g, whether a quarter that lies in one block waits for both groups,
    and where the hand-over of maximum and sum takes its phase from."""
    text = re.sub(r"\s+", " ", source("swa_tc_fwd2.cuh"))
    index, parity = re.search(r"wait_spin\(&sh->o_free((?:\[\w+\])+), ([^;]*)\);", text).groups()
    assert "wait_spin(&sh->ml_empty[qp][quarter], (rec >> kRecUse2 & 1u) ^ 1u);" in text
    assert text.count("mbar_arrive(&sh->ml_empty[qp][slot])") == 1
    if "kRec" in parity:
        return "slot", False
    arrivals = re.findall(r"if \(([^()]*(?:\([^()]*\))?[^()]*)\) mbar_arrive\(&sh->o_free\[(\w+)\]\[slot\]\)", text)
    assert sorted(arrivals) == [("lane == 0", "g1"), ("lane == 0", "g2"), ("lane == g2 || (both && lane == g1)", "lane")]
    head = text[:text.index("mbar_arrive(&sh->o_free[g1][slot])")]
    assert head.rindex("if (both) {") > head.rindex("if constexpr (ONE) {")
    assert "uint32_t free_par = 0xffu;" in text and "free_par ^= fresh << (4 * grp);" in text
    if index == "[grp][e]" and parity == "free_par >> (4 * grp + e) & 1u":
        return "group", False
    assert index == "[0][e]" and parity == "free_par >> e & 1u"
    assert "for (uint32_t h = fresh | alone << 4; h; h &= h - 1) { const int e = (__ffs(h) - 1) ^ 4 * grp;" in text
    assert "alone = rec >> kRecFresh & rec >> kRecEnds & 15u;" in text
    return "group", True


class Clock(dict):
    def join(self, other):
        for k, v in other.items():
            if self.get(k, -1) < v:
                self[k] = v


class Walk:
    """The roles of one CTA over a stream of blocks: `quarters` = (slot, use of the slot, first block, last block)."""

    def __init__(self, o_rule, both_groups):
        self.o_rule, self.both_groups = o_rule, both_groups
        self.at, self.n, self.arrivals, self.waits, self.own, self.wrong = {}, {}, {}, {}, {}, []

    def event(self, role, *after):
        c = Clock(self.at.get(role, {}))
        for a in after:
            if a is not None:
                c.join(a)
        self.n[role] = c[role] = self.n.get(role, -1) + 1
        self.at[role] = c
        return c

    def own_parts(self, role, g, slot):
        return self.own.get((role, g, slot), 0)

    def wait(self, role, bar, k, by):
        """`role` waits for k arrivals on `bar`, all by role `by`."""
        c, a = self.event(role), self.arrivals.get(bar, [])
        known = sum(1 for x in a[:k] if c.get(by, -1) >= x[by])
        if k - known >= 2:
            self.wrong.append(("early", bar, k, known))
        if len(a) > k:
            self.wrong.append(("late", bar, k, len(a)))
        m = known if k - known >= 2 else k
        if m > 0:
            c.join(a[m - 1])
        self.waits.setdefault((bar, k), []).append((role, self.event(role)[role]))

    def arrive(self, role, bar):
        c, a = self.event(role), self.arrivals.setdefault(bar, [])
        for r, n in self.waits.get((bar, len(a)), []):
            if c.get(r, -1) < n:
                self.wrong.append(("late", bar, len(a), r))
        a.append(c)

    def run(self, quarters, n_blocks, nsb, stages, one):
        pv, scores, handed, act, starts = [], [], {}, {}, {}
        for q in quarters:
            starts.setdefault(q[2], []).append(q)
        for n in range(n_blocks):
            for q in starts.get(n, []):
                act[q[0]] = q
            live, g = [q for q in act.values() if q[2] <= n <= q[3]], n & 1
            scores.append(self.event("score", pv[n - nsb] if n >= nsb else None, pv[n - stages] if n >= stages else None))
            masks = []
            for slot in range(4):
                masks.append(self.event(("softmax", g, slot), scores[n]))
                for q in live:
                    if q[0] == slot and q[3] - n < 2:
                        self.wait(("softmax", g, slot), ("ml_empty", q[1] & 1, slot), q[1] >> 1, ("epilogue", slot))
                        masks[-1] = handed[slot, q[1], g] = self.event(("softmax", g, slot))
            for slot, use, first, last in live:
                for h in (g, g ^ 1) if first == last and self.both_groups else (g,) if n - first < 2 else ():
                    k = use if self.o_rule == "slot" else self.own_parts("pv", h, slot)
                    self.wait("pv", ("o_free", h, slot), k, ("epilogue", slot))
            for slot, use, first, last in live:
                if n - first < 2:
                    self.own["pv", g, slot] = self.own_parts("pv", g, slot) + 1
            self.event("pv", *masks)
            pv.append(self.event("pv"))
            for slot, use, first, last in (q for q in live if q[3] == n):
                role, both = ("epilogue", slot), last > first
                other = both or self.o_rule == "slot"               # also arrives for the group of the block before
                if both:
                    self.event(role, handed[slot, use, g ^ 1], pv[n - 1])
                if one and other:
                    self.arrive(role, ("o_free", g ^ 1, slot))
                self.event(role, handed[slot, use, g])
                self.arrive(role, ("ml_empty", use & 1, slot))
                self.event(role, pv[n])
                self.arrive(role, ("o_free", g, slot))
                if not one and other:
                    self.arrive(role, ("o_free", g ^ 1, slot))
        return self.wrong


def plan(th, tw, b, wr, wc, dqk, dv, which=0):
    g = _lib.make_geom(torch.bfloat16, 1, 64, b, th, tw, wr, wc, dqk, dv, 1.0)
    out = (C.c_int32 * 12)()
    return list(out) if _lib.lib.swa_describe_plan(C.byref(g), None, which, out) == 0 else None


def streams(th, tw, b, wr, wc, p, items=12):
    """Quarters and block count of a CTA's first items, for chunks of several heights and items taken in several strides."""
    TW, KR, KW = p[1], p[2], p[3]
    R4, Wtok = 32 // TW, tw * b
    total, strips = -(-th // R4), -(-Wtok // TW)
    halo = max(((x + TW - 1) // b + wc + 1) * b - (x // b - wc) * b for x in range(0, Wtok, TW))
    ncb, unit = -(-halo // KW), next(u for u in range(1, 17) if u * R4 % KR == 0)
    slides = all((i * R4 + R4 - 1 + 2 * wr) // KR < (i + 4) * R4 // KR for i in range(KR))
    for nq in sorted({unit, 2 * unit, 3 * unit, -(-total // unit) * unit}) if slides else [4]:
        for stride in (1, 37, 148):
            quarters, blocks, before = [], 0, 0
            for it in range(0, items * stride, stride):
                r0 = it // strips % -(-total // nq) * nq * R4
                n, h0 = min(nq, -(-(th - r0) // R4)), r0 - wr + KR * (max(0, wr - r0) // KR)
                off, end = r0 - wr - h0, th - 1 - h0
                for i in range(n):
                    first, last = max(i * R4 + off, 0) // KR * ncb, min(i * R4 + off + R4 - 1 + 2 * wr, end) // KR * ncb + ncb - 1
                    quarters.append((before + i & 3, before + i >> 2, blocks + first, blocks + last))
                blocks += (min(n * R4 - 1 + r0 + wr - h0, end) // KR + 1) * ncb
                before += n
            yield quarters, blocks


# one-cell and one-column windows, quarters that one group does alone, items whose borders break the alternation
KNOWN = [(5, 24, 1, 2, 0), (7, 24, 1, 0, 0), (6, 24, 1, 1, 0), (13, 24, 1, 2, 5), (9, 12, 4, 2, 1), (64, 64, 1, 0, 0), (63, 33, 1, 1, 1),
         (81, 65, 1, 1, 0), (9, 93, 1, 7, 0), (83, 127, 1, 3, 1)]


def wrong_waits(o_rule, both_groups, n_random):
    rng, found = random.Random(11), {}
    for t in range(len(KNOWN) + n_random):
        if t < len(KNOWN):
            th, tw, b, wr, wc = KNOWN[t]
            dqk = dv = 64
        else:
            b, th, wr = rng.choice([1, 1, 1, 2, 4, 16]), rng.randint(1, 140), rng.randint(0, 7)
            tw, wc = max(1, rng.randint(1, 100) // b), rng.choice([wr, rng.randint(0, 7)])
            dqk, dv = rng.choice([(64, 64), (64, 64), (32, 32), (128, 128), (128, 64), (64, 128)])
        wr, wc = min(wr, th - 1), min(wc, tw - 1)
        p = plan(th, tw, b, wr, wc, dqk, dv)
        assert p is not None
        for quarters, blocks in streams(th, tw, b, wr, wc, p):
            wrong = Walk(o_rule, both_groups).run(quarters, blocks, p[6], p[5], dqk <= 64 and dv <= 64)
            if wrong:
                found.setdefault((th, tw, b, wr, wc, dqk, dv), wrong)
    return found


def test_every_wait_of_the_forward_kernel_knows_its_phase():
    assert wrong_waits(*rules(), 150) == {}


@pytest.mark.parametrize("o_rule,both_groups,bar,where", [
    ("slot", False, "o_free", [(7, 24, 1, 0, 0), (13, 24, 1, 2, 5), (63, 33, 1, 1, 1)]), ("group", False, "ml_empty", [(81, 65, 1, 1, 0)])])
def test_the_walk_sees_phases_that_are_not_certain(o_rule, both_groups, bar, where):
    """The walk is worth something: waits pass early where the phases of O_g are counted by the uses of the slot, and those of the maxima do
    where a quarter in one block waits for its own group only."""
    found = wrong_waits(o_rule, both_groups, 0)
    for w in where:
        assert any(kind == "early" and b[0] == bar for kind, b, _, _ in found[*w, 64, 64]), w


def test_the_walk_sees_waits_that_come_too_late():
    """... and waits that may never end: the uses of the slot counted, both groups waited for, and the epilogue early for a group without a part."""
    found = wrong_waits("slot", True, 0)
    assert any(kind == "late" and b[0] == "o_free" for kind, b, _, _ in found[7, 24, 1, 0, 0, 64, 64])


def test_the_streams_that_run_on_a_gpu_have_every_kind_of_plan():
    """Keys and values in one ring and in rings of their own (d_qk > 64, three stages), two to four score buffers, one and two resident
    buffers, strips of either width: a change of the planner that loses one of them shows here."""
    plans = [[(dqk, plan(th, tw, b, wr, wc, dqk, dv, which)) for th, tw, b, wr, wc, dqk, dv, _, _ in STREAMS] for which in range(3)]
    assert {p[5] <= 3 for d, p in plans[0] if d > 64} == {True, False}
    assert {p[6] for _, p in plans[0]} >= {3, 4}
    for kernel in plans[1:]:
        assert {p[6] for _, p in kernel} == {2, 3} and {p[7] for _, p in kernel} == {1, 2}
    assert {p[1] for kernel in plans for _, p in kernel} == {8, 16}
