"""CPU model check of the barriers of the split-plane GEMMs (pipeline() in openpv_gb300/csrc/split_gemm.cuh):
the load lane, the MMA lane and the eight epilogue warps of one CTA as coroutines over exact mbarrier semantics,
with a random scheduler between the roles, copies that land in any order and commits that arrive in theirs.

Without a late copy a run must end with every role done, every barrier on a phase boundary and no wait that saw
a barrier more than one phase away.  With copies that are late, every wait is bounded: when nothing can move on,
the limit passes and the waits open at that moment give up.  Whatever is late then, the CTA must not exit with a
copy in flight, unless the wait for that very copy ran out as well.  And a run of many such kernels, of which one
has given up, must end without a limit for each of the others."""
import random

import pytest

EPI = 8


class Cta:
    """One CTA.  late: copies (chunk numbers) that land only after `after` limits have passed.  failed: the run's
    error word on entry, which the load lane reads first and the other waits when they are not over at once."""

    def __init__(self, chunks, stages, seed, late=(), after=1, drain_all=True, failed=False):
        self.chunks, self.stages, self.rnd = chunks, stages, random.Random(seed)
        self.late, self.after, self.drain_all = set(late), after, drain_all
        self.failed = failed
        self.limits = 0  # limits that passed
        self.gen = 0
        self.count, self.pending, self.done = {}, {}, {}
        self.copies, self.held, self.commits, self.aliased = [], [], [], []
        for i in range(stages):
            self.mk(f"full{i}")
            self.mk(f"empty{i}")
        for i in range(2):
            self.mk(f"accFull{i}")
            self.mk(f"accEmpty{i}", EPI)
        self.mk("done")
        self.good = {}
        self.landing_given_up = 0  # waits for a copy in flight that ran out in the drain

    def mk(self, name, n=1):
        self.count[name], self.pending[name], self.done[name] = n, 0, 0

    def arrive(self, name):
        self.pending[name] += 1
        if self.pending[name] == self.count[name]:
            self.pending[name] = 0
            self.done[name] += 1

    def wait(self, name, k):
        """Phase k of a barrier; False when the limit passes first."""
        gen = self.gen
        while True:
            d = self.done[name]
            if not k <= d <= k + 1:
                self.aliased.append((name, k, d))
            if (d & 1) != (k & 1):
                return True
            if self.gen != gen or (self.failed and name != "done"):
                return False
            yield "blocked"

    def drain(self, issued):
        for c in range(max(0, issued - self.stages), issued):
            if not (yield from self.wait(f"full{c % self.stages}", c // self.stages)):
                self.landing_given_up += 1

    def load(self):
        ok, issued = not self.failed, 0
        for c in range(self.chunks if ok else 0):
            s, u = c % self.stages, c // self.stages
            if u and not (yield from self.wait(f"empty{s}", u - 1)):
                ok = False
                break
            (self.held if c in self.late else self.copies).append(f"full{s}")
            issued = c + 1
            yield "step"
        if not ok:
            yield from self.drain(issued)
        yield from self.finish("load", ok)
        if self.drain_all and ok and not all(self.good.values()):
            yield from self.drain(self.chunks)

    def mma(self):
        ok = True
        for c in range(self.chunks):
            s = c % self.stages
            if not (yield from self.wait(f"full{s}", c // self.stages)):
                ok = False
                break
            for h in range(2):
                if c and not (yield from self.wait(f"accEmpty{h}", c - 1)):
                    ok = False
                    break
                self.commits.append(f"accFull{h}")
                yield "step"
            if not ok:
                break
            self.commits.append(f"empty{s}")
        self.commits.append("done")
        yield from self.finish("mma", ok)

    def epilogue(self, w):
        ok = True
        for d in range(2 * self.chunks):
            if not (yield from self.wait(f"accFull{d & 1}", d >> 1)):
                ok = False
                break
            yield "step"
            self.arrive(f"accEmpty{d & 1}")
        yield from self.finish(f"epi{w}", ok)

    def finish(self, role, ok):
        """__syncthreads_and(ok && wait(done)); lanes that do not play a role wait for `done` too."""
        self.good[role] = bool((yield from self.wait("done", 0)) and ok)
        while len(self.good) < 2 + EPI:
            yield "sync"

    def run(self):
        roles = {"load": self.load(), "mma": self.mma()}
        roles.update({f"epi{w}": self.epilogue(w) for w in range(EPI)})
        idle = 0
        while roles:
            if self.limits >= self.after and self.held:
                self.copies, self.held = self.copies + self.held, []
            names = list(roles) + (["copy"] if self.copies else []) + (["commit"] if self.commits else [])
            n = self.rnd.choice(names)
            if n == "copy":
                self.arrive(self.copies.pop(self.rnd.randrange(len(self.copies))))
                idle = 0
                continue
            if n == "commit":
                self.arrive(self.commits.pop(0))
                idle = 0
                continue
            try:
                r = next(roles[n])
            except StopIteration:
                del roles[n]
                idle = 0
                continue
            if r == "step":
                idle = 0
                continue
            idle += 1
            if idle > 40 * (2 + EPI) and not self.copies and not self.commits:
                self.limits += 1  # nothing moves: the waits open now run out
                self.gen += 1
                idle = 0
                assert self.limits < 50, "a wait without a bound"
        return all(self.good.values())

    def in_flight(self):
        return len(self.copies) + len(self.held)


SHAPES = [(c, s) for s in (2, 3) for c in (1, 2, 3, 4, 5, 8)]


@pytest.mark.parametrize("chunks, stages", SHAPES)
def test_every_role_ends_on_a_phase_boundary(chunks, stages):
    for seed in range(20):
        c = Cta(chunks, stages, seed)
        assert c.run() and c.limits == 0
        assert not c.aliased and not any(c.pending.values()) and not c.in_flight() and not c.commits


@pytest.mark.parametrize("chunks, stages", SHAPES)
def test_no_copy_in_flight_at_exit(chunks, stages):
    """One copy late by a limit or two, at every place, among the last ones (all issued by then) as well."""
    for late in range(chunks):
        for after in (1, 2):
            for seed in range(5):
                c = Cta(chunks, stages, seed, {late}, after)
                assert not c.run()
                assert not c.commits and c.in_flight() <= c.landing_given_up
                if after == 1:
                    assert c.in_flight() == 0, (late, seed)


@pytest.mark.parametrize("chunks, stages", SHAPES)
def test_a_failed_run_ends_promptly(chunks, stages):
    """Copies that never land, from the first of forty kernels on: one limit for its waits and one for each copy it
    has in flight, none for the kernels after it -- and one and more for each where the error word is not read."""
    def run(reads):
        limits, failed = 0, False
        for k in range(40):
            c = Cta(chunks, stages, k, range(chunks), 1 << 30, failed=failed and reads)
            failed = not c.run() or failed
            limits += c.limits
            assert not c.commits and c.in_flight() <= c.landing_given_up
        return limits
    assert run(True) <= 1 + stages
    assert run(False) >= 40


def test_a_drain_by_the_load_lane_alone_is_caught():
    """The load lane waiting for its copies only when its own wait gave up: a late copy among the last `stages`
    ones outlives the CTA, and the model finds it."""
    found = []
    for chunks, stages in SHAPES:
        c = Cta(chunks, stages, 1, {chunks - 1}, 2, drain_all=False)
        assert not c.run()
        found.append(c.in_flight() > c.landing_given_up)
    assert all(found), found
