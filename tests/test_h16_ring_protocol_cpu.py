"""Model check of the 16-bit ring kernel's accumulators (kami_b200/csrc/h16_ring.cu)
on the CPU: two copying warps that join one barrier per chunk, the thread that
issues a group's MMAs, and the warps that store C, over mbarriers that only tell
the parity of a phase, MMAs that run some time after they are issued, problems of
up to 64 columns (two accumulators) and of more (both at once) in any order; and
the form for large problems, whose two sets of storing warps take turns.  No
accumulator may be written while it is read or before it has been, every problem
must be stored from its own product, and nobody may wait for good.  Without the
wait for both accumulators the check must fail."""
import random

import pytest

RECS = 16


class Bar:
    def __init__(self, count):
        self.count, self.pending, self.phase = count, count, 0

    def arrive(self):
        self.pending -= 1
        assert self.pending >= 0
        if self.pending == 0:
            self.pending, self.phase = self.count, self.phase + 1

    def passed(self, parity):
        return self.phase % 2 != parity


def simulate(rng, problems, slots, two, wide_wait=True):
    """problems: (columns, chunks) each"""
    slots = min(slots, RECS)
    chunks = [(p, c == 0, c == n - 1) for p, (_, n) in enumerate(problems) for c in range(n)]
    full = [Bar(3) for _ in range(RECS)]  # two copying warps and the record
    empty = [Bar(1) for _ in range(RECS)]
    accf, acce = [Bar(2) for _ in range(2)], [Bar(4) for _ in range(2)]
    slot_of = [None] * slots         # the chunk whose bytes a slot holds
    landed = [0] * len(chunks)
    owner = [None] * 4               # problem in each 64 columns of the accumulators, once written
    unread = [0] * 4                 # warps that still have to read them
    grec = [None, None]
    pipe = []                        # the tensor core: what is left, in order
    stored = [0] * len(problems)

    def columns(p, b):
        if two:
            return [2 * b, 2 * b + 1][:1 + (problems[p][0] > 64)]
        return [0, 1] if problems[p][0] > 64 else [b]

    def copier(which):
        for j in range(len(chunks)):
            dep = j - slots
            if dep >= 0:
                while not empty[dep % RECS].passed((dep // RECS) & 1):
                    yield
                assert slot_of[j % slots] in (dep, j)
            slot_of[j % slots] = j
            yield
            landed[j] += 1
            full[j % RECS].arrive()
            if which == 0:
                full[j % RECS].arrive()  # the record
            yield

    def issuer():
        turn, wide = 0, False
        for j, (p, first, last) in enumerate(chunks):
            b = turn & 1
            while not full[j % RECS].passed((j // RECS) & 1):
                yield
            assert landed[j] == 2 and slot_of[j % slots] == j
            if first:
                now = problems[p][0] > 64 and not two
                if turn >= 2:
                    while not acce[b].passed(((turn >> 1) - 1) & 1):
                        yield
                if turn >= 1 and (now or wide) and wide_wait:
                    while not acce[b ^ 1].passed(((turn - 1) >> 1) & 1):
                        yield
                wide = now
                assert grec[b] is None, "record overwritten before it was read"
                grec[b] = [p, 4]
            pipe.append(("mma", p, b, j, first))
            yield
            pipe.append(("commit", empty[j % RECS]))
            if last:
                pipe.append(("commit", accf[b]))
                accf[b].arrive()
                turn += 1
            yield

    def storer(half, _):
        for turn in range(half if two else 0, len(problems), 2 if two else 1):
            b = turn & 1
            while not accf[b].passed((turn >> 1) & 1):
                yield
            p = grec[b][0]
            assert p == turn
            for c in columns(p, b):
                assert owner[c] == p
                yield
                assert owner[c] == p, "accumulator overwritten while it is read"
                unread[c] -= 1
            stored[p] += 1
            grec[b][1] -= 1
            if grec[b][1] == 0:
                grec[b] = None
            acce[b].arrive()
            yield

    sets = (0, 1) if two else (0,)
    roles = [copier(0), copier(1), issuer()] + [storer(h, q) for h in sets for q in range(4)]
    speed = [rng.choice((1.0, 0.5, 0.05)) for _ in roles] + [rng.choice((1.0, 0.3, 0.03))]
    live, idle = set(range(len(roles))), 0
    while live or pipe:
        idle += 1
        assert idle < 40000, "no progress"
        if pipe and rng.random() < speed[-1]:
            idle = 0
            what = pipe.pop(0)
            if what[0] == "commit":
                what[1].arrive()
            else:
                _, p, b, j, first = what
                assert slot_of[j % slots] == j, "operands overwritten before the MMA"
                for c in columns(p, b):
                    assert unread[c] == 0 if first else owner[c] == p, "accumulator overwritten"
                    owner[c], unread[c] = p, 4
        if live:
            r = rng.choice(sorted(live))
            if rng.random() < speed[r]:
                before = (sum(stored), sum(landed), len(pipe))
                try:
                    next(roles[r])
                except StopIteration:
                    live.discard(r)
                    idle = 0
                if (sum(stored), sum(landed), len(pipe)) != before:
                    idle = 0
    assert stored == [4] * len(problems)


def _problems(rng, kind):
    n = rng.randrange(1, 50)
    cols = {"narrow": (16, 64), "wide": (80, 128), "mixed": (16, 128, 64, 65)}[kind]
    return [(rng.choice(cols), rng.choice((1, 1, 2))) for _ in range(n)]


@pytest.mark.parametrize("kind", ["narrow", "wide", "mixed"])
@pytest.mark.parametrize("slots", [1, 2, 5, 16])
@pytest.mark.parametrize("two", [False, True])
def test_accumulators(kind, slots, two):
    rng = random.Random(f"{kind} {slots} {two}")
    for _ in range(12):
        simulate(rng, _problems(rng, kind), slots, two)


def test_needs_the_wait_for_both(kind="mixed"):
    rng = random.Random(1)
    with pytest.raises(AssertionError, match="overwritten"):
        for _ in range(50):
            simulate(rng, _problems(rng, kind), 5, False, wide_wait=False)
