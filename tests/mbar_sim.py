"""One CTA's roles as coroutines over exact mbarrier semantics, with copies that may be late and waits that are
bounded: when nothing can move on, the limit passes and the waits open at that moment give up.

A wait for phase k tests parity k & 1 and passes once the barrier has completed a phase of the other parity; a
barrier completes a phase when its expected arrivals are in.  Copies land in any order, commits in issue order."""
import random


class Cta:
    def __init__(self, seed, late=(), after=1):
        """late: keys of the copies that land only after `after` limits have passed."""
        self.rnd = random.Random(seed)
        self.late, self.after = set(late), after
        self.limits = self.gen = 0
        self.count, self.pending, self.done = {}, {}, {}
        self.copies, self.held, self.commits, self.aliased = [], [], [], []
        self.given_up_landing = 0  # waits for a copy in flight that ran out in a drain

    def mk(self, name, n=1):
        self.count[name], self.pending[name], self.done[name] = n, 0, 0

    def arrive(self, name):
        self.pending[name] += 1
        assert self.pending[name] <= self.count[name], name
        if self.pending[name] == self.count[name]:
            self.pending[name] = 0
            self.done[name] += 1

    def test(self, name, k):
        d = self.done[name]
        if not k <= d <= k + 1:
            self.aliased.append((name, k, d))
        return (d & 1) != (k & 1)

    def wait(self, name, k):
        """Phase k of a barrier; False when the limit passes first."""
        gen = self.gen
        while not self.test(name, k):
            if self.gen != gen:
                return False
            yield "blocked"
        return True

    def copy(self, key, name):
        (self.held if key in self.late else self.copies).append(name)

    def land(self, ring, slots, issued):
        """The last copies of a ring of `slots` barriers, `issued` in all."""
        for c in range(max(0, issued - slots), issued):
            if not (yield from self.wait(f"{ring}{c % slots}", c // slots)):
                self.given_up_landing += 1

    def in_flight(self):
        return len(self.copies) + len(self.held)

    def play(self, roles):
        idle = 0
        while roles:
            if self.limits >= self.after and self.held:
                self.copies, self.held = self.copies + self.held, []
            n = self.rnd.choice(list(roles) + (["copy"] if self.copies else []) + (["commit"] if self.commits else []))
            if n == "copy":
                self.arrive(self.copies.pop(self.rnd.randrange(len(self.copies))))
                idle = 0
            elif n == "commit":
                self.arrive(self.commits.pop(0))
                idle = 0
            else:
                try:
                    r = next(roles[n])
                except StopIteration:
                    del roles[n]
                    r = "step"
                idle = 0 if r == "step" else idle + 1
            if idle > 60 * len(roles) + 60 and not self.copies and not self.commits:
                self.limits += 1  # nothing moves: the waits open now run out
                self.gen += 1
                idle = 0
                assert self.limits < 80, "a wait without a bound"
