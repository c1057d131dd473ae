"""Chunked DFA walks by entry states (csrc/dfa_chunks.cuh), its rules written out on the CPU and
held against the serial walk: collapse to a few entry states or not at all, one walk per entry
state on to the next chunk's entry position, latches that stop later chunks at any time, and
the fix-up that follows the records and walks the gaps. Small constants stand for the device's
(entry states, bytes between two looks at the latch, bytes of a first chunk's prefix)."""

from __future__ import annotations

import numpy as np
import pytest

MEET, LISTED = 4, 32  # kMeetBytes; members up to which a set's steps are not budgeted


class Model:
    def __init__(self, trans, accept, start, data, chunks, entries, prefix, poll, overlap, budget,
                 rng):
        self.t, self.acc, self.start, self.x = trans, accept, start, data
        n = len(data)
        self.bounds = [(k * n // chunks, (k + 1) * n // chunks) for k in range(chunks)]
        self.entries, self.prefix, self.poll = entries, prefix, poll
        self.overlap, self.budget, self.rng = overlap, budget, rng
        self.latch = 1 << 30

    def span(self, s, a, b):
        """(state at b or at the first accept, that accept's position or -1)"""
        for q in range(a, b):
            s = int(self.t[s, self.x[q]])
            if self.acc[s]:
                return s, q + 1
        return s, -1

    def collapse(self, b, e):
        members, left = np.arange(self.t.shape[0]), self.budget
        if e <= b:
            return -1, members
        pos = b
        while members.size > self.entries and pos < e:
            k = 1 if pos == b and members.size > LISTED else min(MEET, e - pos)
            if members.size > LISTED:
                if left < 0:
                    return -1, members
                left -= members.size * k
            for c in self.x[pos:pos + k]:
                members = self.t[members, c]
            members = np.unique(members)
            pos += k
        return (pos, members) if members.size <= self.entries else (-1, members)

    def may_stop(self, index):
        return self.latch < index and self.rng.random() < 0.7

    def first_launch(self):
        self.rec = []
        order = self.rng.permutation(len(self.bounds))
        done = {}
        for i in order:
            b, e = self.bounds[i]
            if i == 0:
                p, acc, s = min(e, self.prefix), -1, self.start
                if self.acc[s]:
                    acc = 0
                else:
                    s, acc = self.span(s, 0, p)
                if acc >= 0:
                    self.latch = min(self.latch, 0)
                done[i] = dict(p=p, at=p, entry=[s], exit=[s], acc=[acc], done=p)
            elif self.may_stop(i):
                done[i] = dict(p=-2, at=-1, entry=[], exit=[], acc=[], done=0)
            else:
                p, m = self.collapse(b, e)
                m = m.tolist() if p >= 0 else []
                done[i] = dict(p=p, at=p, entry=m, exit=list(m), acc=[-1] * len(m),
                               done=max(p, 0))
        self.rec = [done[i] for i in range(len(self.bounds))]

    def target(self, i):
        cap = min(len(self.x), self.bounds[i][1] + self.overlap)
        for r in self.rec[i + 1:]:
            if r["at"] >= 0:
                return min(cap, r["at"])
        return cap

    def walk_launch(self):
        for i in self.rng.permutation(len(self.rec)):
            r = self.rec[i]
            if r["p"] < 0:
                continue
            q, target = r["p"], self.target(i)
            while q < target and not all(a >= 0 for a in r["acc"]):
                if self.may_stop(i):
                    r["p"] = -2
                    break
                to = min(target, q + self.poll)
                for g, a in enumerate(r["acc"]):
                    if a < 0:
                        r["exit"][g], r["acc"][g] = self.span(r["exit"][g], q, to)
                q = to
            if all(a >= 0 for a in r["acc"]) and r["acc"]:
                self.latch = min(self.latch, i)
            r["done"] = q

    def fixup(self):
        known, pos, s = False, 0, 0
        for r in self.rec:
            if r["p"] < 0:
                continue
            if not known:
                known, s = True, r["entry"][0]
            elif pos < r["p"]:
                s, acc = self.span(s, pos, r["p"])
                if acc >= 0:
                    return acc
            elif pos > r["p"]:
                continue
            pos = r["p"]
            if s not in r["entry"]:
                continue
            g = r["entry"].index(s)
            if r["acc"][g] >= 0:
                return r["acc"][g]
            s, pos = r["exit"][g], r["done"]
        return self.span(s, pos, len(self.x))[1]

    def verdict(self):
        self.first_launch()
        self.walk_launch()
        return self.fixup()


def _dfa(rng, n, kind, accepts):
    t = rng.integers(0, n, size=(n, 7))
    if kind == "permuting":
        t = np.stack([rng.permutation(n) for _ in range(7)], axis=1)
    elif kind == "group":  # shrinks to a group that is permuted for good
        g = min(n, 6)
        t = rng.integers(0, g, size=(n, 7))
        for c in range(7):
            t[:g, c] = rng.permutation(g)
    accept = np.zeros(n, bool)
    accept[rng.permutation(n)[:accepts]] = True
    return t, accept


@pytest.mark.parametrize("kind", ["random", "permuting", "group"])
@pytest.mark.parametrize("n", [1, 3, 40, 150])
def test_records_lead_to_the_serial_verdict(kind, n):
    rng = np.random.default_rng(n)
    seen = set()
    for case in range(150):
        t, accept = _dfa(rng, n, kind, int(rng.integers(0, 2 if n > 3 else 1) * (case % 3 > 0)))
        x = rng.integers(0, 7, int(rng.integers(1, 700)))
        start = int(rng.integers(0, n))
        m = Model(t, accept, start, x, chunks=int(rng.integers(1, 9)),
                  entries=int(rng.choice([2, 5, 16])), prefix=int(rng.choice([4, 50])),
                  poll=int(rng.choice([3, 16])), overlap=int(rng.choice([0, 5, 1 << 20])),
                  budget=int(rng.choice([0, 400, 1 << 20])), rng=rng)
        want = 0 if accept[start] else m.span(start, 0, len(x))[1]
        assert m.verdict() == want
        seen |= {r["p"] if r["p"] < 0 else 0 for r in m.rec}
    assert 0 in seen and (n < 40 or -1 in seen)


def test_some_chunks_are_stopped():
    rng = np.random.default_rng(5)
    stopped = 0
    for _ in range(50):
        t, accept = _dfa(rng, 60, "random", 3)
        x = rng.integers(0, 7, 600)
        m = Model(t, accept, 0, x, 8, 4, 30, 8, 1 << 20, 1 << 20, rng)
        want = 0 if accept[0] else m.span(0, 0, len(x))[1]
        assert m.verdict() == want
        stopped += sum(r["p"] == -2 for r in m.rec)
    assert stopped > 20
