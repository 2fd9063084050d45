"""Model check of the ring kernels' protocol (kami_b200/csrc/ring.cuh) on the
CPU: copying warps place chunks of random size by the schedule the host works
out, each taking its own chunks, and computing groups pass them in order, over
mbarriers that only tell the parity of a phase.  No wait may pass before what
it waits for, none may be missed for good, and no bytes may be overwritten
that are still read."""
import random

import pytest

RECS = 32


def place(sizes, ring, most):
    """ring::Placer: (at, dep, land) of every chunk."""
    spans, head, gone, out = [], 0, -1, []
    for j, b in enumerate(sizes):
        at = 0 if head + b > ring else head
        gone = max(gone, j - RECS)
        q = gone + 1
        while q < j and at < head and spans[q][0] >= head:
            q += 1
        while q < j and spans[q][0] < at + b and at < spans[q][1]:
            gone = q
            q += 1
        head = at + b
        spans.append((at, head))
        land, fly = j - 1, b
        while land > gone and fly < most:
            fly += sizes[land]
            land -= 1
        out.append((at, gone, land))
    return out


class Bar:
    """phases completed so far, and arrivals pending in the current one"""

    def __init__(self, count):
        self.count, self.pending, self.phase = count, count, 0

    def arrive(self):
        self.pending -= 1
        assert self.pending >= 0
        if self.pending == 0:
            self.pending, self.phase = self.count, self.phase + 1

    def passed(self, parity):
        return self.phase % 2 != parity


def simulate(sizes, ring, most, copiers, groups, rng):
    n = len(sizes)
    sched = place(sizes, ring, most)
    for j, (at, dep, land) in enumerate(sched):
        assert at + sizes[j] <= ring and j - RECS <= dep <= land < j
        for i in range(dep + 1, j):
            assert sched[i][0] + sizes[i] <= at or at + sizes[j] <= sched[i][0], "bytes still read are overwritten"
    full = [Bar(1) for _ in range(RECS)]
    empty = [Bar(groups) for _ in range(RECS)]
    landed, passed_by = [False] * n, [0] * n
    flying = []

    def copier(cw):
        gone = -1
        for j in range(cw, n, copiers):
            _, dep, land = sched[j]
            while gone < dep:
                to = min(dep, gone + RECS)
                while not empty[to % RECS].passed((to // RECS) & 1):
                    yield
                assert all(p == groups for p in passed_by[:to + 1]), "chunk still in use"
                gone = to
            if land > gone:
                s, parity = land % RECS, (land // RECS) & 1
                while not (empty[s].passed(parity) or full[s].passed(parity)):
                    yield
                assert landed[land]
            flying.append(j)
            yield

    def group():
        for j in range(n):
            while not full[j % RECS].passed((j // RECS) & 1):
                yield
            assert landed[j] and not any(landed[j + RECS:j + RECS + 1])
            for _ in range(rng.choice((0, 0, 1, 8))):
                yield
            passed_by[j] += 1
            empty[j % RECS].arrive()
            yield

    roles = [copier(c) for c in range(copiers)] + [group() for _ in range(groups)]
    speed = [rng.choice((1.0, 1.0, 0.2, 0.02)) for _ in roles]
    live, idle = set(range(len(roles))), 0
    while live:
        idle += 1
        assert idle < 200000, "no progress"
        r = rng.choice(sorted(live))
        if rng.random() < speed[r]:
            before = (sum(passed_by), len(flying))
            try:
                next(roles[r])
            except StopIteration:
                live.discard(r)
                idle = 0
            if (sum(passed_by), len(flying)) != before:
                idle = 0
        while flying and rng.random() < 0.3:
            j = flying.pop(rng.randrange(len(flying)))
            landed[j] = True
            full[j % RECS].arrive()


@pytest.mark.parametrize("sizes", ["small", "large", "mixed", "one size"])
@pytest.mark.parametrize("most", [1, 64, 10 ** 6])
def test_ring_protocol(sizes, most):
    rng = random.Random(f"{sizes} {most}")
    for _ in range(4):
        one = rng.randrange(1, 70)
        draw = {"small": lambda: rng.randrange(1, 6), "large": lambda: rng.randrange(40, 75),
                "mixed": lambda: rng.choice((1, 2, 3, 20, 60)), "one size": lambda: one}[sizes]
        simulate([draw() for _ in range(rng.randrange(1, 160))], 224, most, 4, rng.choice((1, 4, 16)), rng)
