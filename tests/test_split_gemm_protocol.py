"""CPU model check of the barriers of the split-plane GEMMs (pipeline() in openpv_gb300/csrc/split_gemm.cuh):
the load lane, the MMA lane and the eight epilogue warps of one CTA as coroutines over exact mbarrier semantics,
with a random scheduler between the roles, copies that land in any order and commits that arrive in theirs.

Without a late copy a run must end with every role done, every barrier on a phase boundary and no wait that saw
a barrier more than one phase away.  With copies that are late, every wait is bounded: when nothing can move on,
the limit passes and the waits open at that moment give up.  Whatever is late then, the CTA must not exit with a
copy in flight, unless the wait for that very copy ran out as well.  And a run of many such kernels, of which one
has given up, must end without a limit for each of the others."""
import pytest

from tests.mbar_sim import Cta

EPI = 8


class Pipeline(Cta):
    """failed: the run's error word on entry, which the load lane reads first and the other waits when they are not
    over at once."""

    def __init__(self, chunks, stages, seed, late=(), after=1, drain_all=True, failed=False):
        super().__init__(seed, late, after)
        self.chunks, self.stages, self.drain_all, self.failed = chunks, stages, drain_all, failed
        for i in range(stages):
            self.mk(f"full{i}")
            self.mk(f"empty{i}")
        for i in range(2):
            self.mk(f"accFull{i}")
            self.mk(f"accEmpty{i}", EPI)
        self.mk("done")
        self.good = {}

    def wait(self, name, k):
        if self.failed and name != "done":
            yield "step"
            return self.test(name, k)
        return (yield from super().wait(name, k))

    def drain(self, issued):
        yield from self.land("full", self.stages, issued)

    def load(self):
        ok, issued = not self.failed, 0
        for c in range(self.chunks if ok else 0):
            s, u = c % self.stages, c // self.stages
            if u and not (yield from self.wait(f"empty{s}", u - 1)):
                ok = False
                break
            self.copy(c, f"full{s}")
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
        self.play(roles)
        return all(self.good.values())


SHAPES = [(c, s) for s in (2, 3) for c in (1, 2, 3, 4, 5, 8)]


@pytest.mark.parametrize("chunks, stages", SHAPES)
def test_every_role_ends_on_a_phase_boundary(chunks, stages):
    for seed in range(20):
        c = Pipeline(chunks, stages, seed)
        assert c.run() and c.limits == 0
        assert not c.aliased and not any(c.pending.values()) and not c.in_flight() and not c.commits


@pytest.mark.parametrize("chunks, stages", SHAPES)
def test_no_copy_in_flight_at_exit(chunks, stages):
    """One copy late by a limit or two, at every place, among the last ones (all issued by then) as well."""
    for late in range(chunks):
        for after in (1, 2):
            for seed in range(5):
                c = Pipeline(chunks, stages, seed, {late}, after)
                assert not c.run()
                assert not c.commits and c.in_flight() <= c.given_up_landing
                if after == 1:
                    assert c.in_flight() == 0, (late, seed)


@pytest.mark.parametrize("chunks, stages", SHAPES)
def test_a_failed_run_ends_promptly(chunks, stages):
    """Copies that never land, from the first of forty kernels on: one limit for its waits and one for each copy it
    has in flight, none for the kernels after it -- and one and more for each where the error word is not read."""
    def run(reads):
        limits, failed = 0, False
        for k in range(40):
            c = Pipeline(chunks, stages, k, range(chunks), 1 << 30, failed=failed and reads)
            failed = not c.run() or failed
            limits += c.limits
            assert not c.commits and c.in_flight() <= c.given_up_landing
        return limits
    assert run(True) <= 1 + stages
    assert run(False) >= 40


def test_a_drain_by_the_load_lane_alone_is_caught():
    """The load lane waiting for its copies only when its own wait gave up: a late copy among the last `stages`
    ones outlives the CTA, and the model finds it."""
    found = []
    for chunks, stages in SHAPES:
        c = Pipeline(chunks, stages, 1, {chunks - 1}, 2, drain_all=False)
        assert not c.run()
        found.append(c.in_flight() > c.given_up_landing)
    assert all(found), found
