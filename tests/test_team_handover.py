"""Schedule-fuzzing model of the decode kernel's teams (csrc/megakernel.cu, team_rows and epilogue_role): teams of four warps that sum
the rows of ring stages, and one warp that takes the sums over in groups of tasks.

Ring.  A slot has a `full` barrier (one arrival, the producer's) and an `empty` one (one arrival per consumer warp).  In a phase whose
stages hold one task each, a stage belongs to the team slot % teams: only its warps wait for it, and each gives it back `teams` times.
In every other phase every warp waits on every stage and gives it back once.  All warps meet between phases.  A waiter only learns the
parity of the last completed phase of a barrier, so the model keeps barriers that answer by parity alone.

Hand-over.  Two buffers of `group` tasks in turn.  A warp waits for the buffer to be empty before its first task of a group, writes its
sum, arrives on the buffer's `full` barrier (4 * group arrivals); the epilogue warp arrives for the tasks that a phase's last group
lacks, waits, reads all members' sums and empties the buffer.

Bulk copies land in any order.  The model fails when a stage is read that does not hold the expected fill or is refilled under a reader, when a sum is overwritten
before it was read or read before it was written, and when everybody waits.
"""
import random

import pytest

MEMBERS = 4


class ProtocolError(AssertionError):
    pass


class MBarrier:
    def __init__(self, arrivals):
        self.arrivals, self.pending, self.completed = arrivals, arrivals, 0

    def arrive(self, count=1):
        if count > self.pending:
            raise ProtocolError("more arrivals than a phase of the barrier has")
        self.pending -= count
        if self.pending == 0:
            self.completed += 1
            self.pending = self.arrivals

    def passed(self, parity):
        return ((self.completed - 1) & 1) == parity


class Model:
    def __init__(self, teams, slots, group, phases):
        self.teams, self.slots, self.group, self.phases = teams, slots, group, phases
        self.warps = teams * MEMBERS
        self.full = [MBarrier(1) for _ in range(slots)]
        self.empty = [MBarrier(self.warps) for _ in range(slots)]
        self.part_full = [MBarrier(MEMBERS * group) for _ in range(2)]
        self.part_empty = [MBarrier(1) for _ in range(2)]
        self.data = [None] * slots
        self.readers = [set() for _ in range(slots)]
        self.part = [{} for _ in range(2)]
        self.met = [0] * len(phases)
        self.flight, self.issued = [], False

    def producer(self):
        n = 0
        for _, stages, _, _ in self.phases:
            for _ in range(stages):
                slot, parity = n % self.slots, (n // self.slots) & 1
                while not self.empty[slot].passed(parity ^ 1):
                    yield "wait"
                if self.readers[slot]:
                    raise ProtocolError(f"fill {n} overwrites slot {slot} under {sorted(self.readers[slot])}")
                self.data[slot] = None
                self.flight.append(n)
                yield "copy"
                n += 1
        self.issued = True

    def copies(self, rng):  # land in any order
        while self.flight or not self.issued:
            if not self.flight:
                yield "wait"
                continue
            n = self.flight.pop(rng.randrange(len(self.flight)))
            self.data[n % self.slots] = n
            self.full[n % self.slots].arrive()
            yield "land"

    def take(self, warp, n):
        slot = n % self.slots
        while not self.full[slot].passed((n // self.slots) & 1):
            yield "wait"
        self.readers[slot].add(warp)
        for _ in range(2):
            if self.data[slot] != n:
                raise ProtocolError(f"warp {warp} expected fill {n} in slot {slot}, found {self.data[slot]}")
            yield "read"
        self.readers[slot].discard(warp)

    def consumer(self, warp):
        team, member = warp // MEMBERS, warp % MEMBERS
        first, groups = 0, 0  # fills and groups of the phases before
        for p, (kind, stages, per_stage, last) in enumerate(self.phases):
            self.met[p] += 1
            while self.met[p] < self.warps:  # the barrier between phases
                yield "wait"
            tasks = 0 if kind == "all" else (stages - 1) * per_stage + last
            entered = None

            def deliver(task):
                nonlocal entered
                at = groups + task // self.group
                if entered != at:
                    while not self.part_empty[at & 1].passed(((at >> 1) & 1) ^ 1):
                        yield "wait"
                    entered = at
                key = (task % self.group, member)
                if key in self.part[at & 1]:
                    raise ProtocolError(f"warp {warp}: sum {key} of group {at} is overwritten")
                self.part[at & 1][key] = (p, task)
                yield "write"
                self.part_full[at & 1].arrive()

            for i in range(stages):
                n = first + i
                mine = range(i * per_stage, min((i + 1) * per_stage, tasks))
                if kind in ("owned", "by fill"):
                    if (n % self.slots if kind == "owned" else n) % self.teams != team:
                        continue
                    times = self.teams
                else:
                    times, mine = 1, [t for t in mine if kind != "all" and t % self.teams == team]
                yield from self.take(warp, n)
                self.empty[n % self.slots].arrive(times)
                for t in mine:
                    yield from deliver(t)
            first += stages
            groups += -(-tasks // self.group)

    def epilogue(self):
        at = 0
        for p, (kind, stages, per_stage, last) in enumerate(self.phases):
            tasks = 0 if kind == "all" else (stages - 1) * per_stage + last
            for g in range(-(-tasks // self.group)):
                here = min(self.group, tasks - g * self.group)
                if here < self.group:
                    self.part_full[at & 1].arrive(MEMBERS * (self.group - here))
                while not self.part_full[at & 1].passed((at >> 1) & 1):
                    yield "wait"
                want = {(t, m): (p, g * self.group + t) for t in range(here) for m in range(MEMBERS)}
                yield "read"
                if self.part[at & 1] != want:
                    raise ProtocolError(f"group {at}: not the sums of its tasks")
                self.part[at & 1] = {}
                self.part_empty[at & 1].arrive()
                at += 1


def run(model, seed, bias):
    rng = random.Random(seed)
    procs = {"p": model.producer(), "c": model.copies(rng), "e": model.epilogue(), **{w: model.consumer(w) for w in range(model.warps)}}
    fast, slow = rng.sample(list(procs), 2)
    idle = 0
    while procs:
        keys = list(procs)
        if idle > 2000:  # a long wait may only mean that the slow one was not drawn
            k = rng.choice(keys)
        elif fast in procs and rng.random() < bias:
            k = fast
        else:
            k = rng.choice(([x for x in keys if x != slow] or keys) if rng.random() < bias else keys)
        try:
            op = next(procs[k])
        except StopIteration:
            del procs[k]
            idle = 0
            continue
        idle = idle + 1 if op == "wait" else 0
        if idle > 20000:
            raise ProtocolError("everybody waits")


def phases_of(rng, teams, slots):
    out = []
    for _ in range(7):
        kind = rng.choice(["owned", "shared", "all"] if slots % teams == 0 else ["shared", "all"])
        per_stage = 1 if kind != "shared" else rng.choice([1, 2, 3, 7])
        out.append((kind, rng.randint(1, 3 * slots), per_stage, rng.randint(1, per_stage)))
    return out


@pytest.mark.parametrize("teams,slots", [(2, 6), (2, 4), (2, 5), (3, 6), (3, 4), (2, 2)])
@pytest.mark.parametrize("group", [8, 4])
def test_every_schedule_hands_every_sum_over_once(teams, slots, group):
    for seed in range(8):
        phases = phases_of(random.Random(100 + seed), teams, slots)
        for bias in (0.0, 0.8, 0.97):
            run(Model(teams, slots, group, phases), seed, bias)


def test_slots_that_change_teams_are_not_safe():
    """Were stages given to the teams by their fill's number and the slots not a multiple of the teams, a slot's fills would go to
    different teams in turn: one of them can wait for a fill while the one before it has not landed, and takes the parity of an older
    one for it.  The kernel shares the stages of such a ring between the teams instead."""
    caught = 0
    for seed in range(40):
        for bias in (0.0, 0.8, 0.97):
            try:
                run(Model(3, 4, 8, [("by fill", 24, 1, 1)] * 3), seed, bias)
            except ProtocolError:
                caught += 1
    assert caught > 0
