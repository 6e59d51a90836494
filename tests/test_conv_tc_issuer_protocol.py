"""CPU model check of the tensor-core delivery's barriers (conv_tf32x3_kernel in openpv_gb300/csrc/deliver_tc.cu) with
its MMA warp: the split row's slot and phase and the weight tile's carried along by additions, the next tile's
barrier probed in the middle of a tile's MMAs, a wait only where the probe found nothing; and with copies that are
late, after which every role must end by the abort flag or its own limit and the CTA must not exit with a copy in
flight, unless the wait for that very copy ran out as well."""
import pytest

from tests.mbar_sim import Cta


class Conv(Cta):
    """R target rows per unit, NS split-row slots, NR raw-row slots, NB weight-tile slots, KX x KY patch, nFC source
    chunks, units of this CTA.  drain_all False: the producer waits for its copies only when it gave up itself."""

    def __init__(self, R, NS, NR, NB, KX, KY, nFC, units, seed, late=(), after=1, drain_all=True, carry=True):
        super().__init__(seed, late, after)
        self.p = R, NS, NR, NB, KX, KY, nFC, units
        self.drain_all, self.carry = drain_all, carry
        self.abort, self.left = False, 0
        for i in range(NR):
            self.mk(f"rawFull{i}")
            self.mk(f"rawEmpty{i}", 4)
        for i in range(NS):
            self.mk(f"aReady{i}", 4)
            self.mk(f"aEmpty{i}")
        for i in range(NB):
            self.mk(f"bFull{i}")
            self.mk(f"bEmpty{i}")
        for i in range(2):
            self.mk(f"chainFull{i}")
            self.mk(f"chainEmpty{i}", 4)
        self.mk("done")
        self.per_chain = max(1, min(KY, (7 + KX - 1) // KX))
        self.chains = (nFC * KY + self.per_chain - 1) // self.per_chain

    def bounded(self, name, k):
        """wait_or_abort / warp_wait: a look, the abort flag, then the wait; running out raises the flag."""
        if self.test(name, k):
            return True
        if self.abort:
            return False
        ok = yield from self.wait(name, k)
        if not ok:
            self.abort = True
        return ok

    def producer(self):
        R, NS, NR, NB, KX, KY, nFC, units = self.p
        ca = cb = 0

        def load_a():
            nonlocal ca
            if ca >= NR and not (yield from self.bounded(f"rawEmpty{ca % NR}", ca // NR - 1)):
                return False
            self.copy(("a", ca), f"rawFull{ca % NR}")
            ca += 1
            yield "step"
            return True

        def load_b():
            nonlocal cb
            if cb >= NB and not (yield from self.bounded(f"bEmpty{cb % NB}", cb // NB - 1)):
                return False
            self.copy(("b", cb), f"bFull{cb % NB}")
            cb += 1
            yield "step"
            return True

        ok = True
        for _ in range(units * nFC):
            for _ in range(R - 1):
                ok = ok and (yield from load_a())
            for _ in range(KY):
                ok = ok and (yield from load_a())
                for _ in range(KX):
                    ok = ok and (yield from load_b())
        if not self.drain_all and not ok:
            yield from self.drain(ca, cb)
        self.left += 1
        while self.left < 10:
            yield "sync"
        if self.drain_all and self.abort:
            yield from self.drain(ca, cb)

    def drain(self, ca, cb):
        _, _, NR, NB, *_ = self.p
        yield from self.land("rawFull", NR, ca)
        yield from self.land("bFull", NB, cb)

    def mma(self):
        R, NS, NR, NB, KX, KY, nFC, units = self.p
        cc = slot = use = d = tile = 0  # chains; split row `use * NS + slot`; weight tile `tile * NB + d`
        seen = False
        ok = True

        def row(ahead):
            sl, u = slot + ahead, use
            if sl >= NS:
                sl, u = sl - NS, u + 1
            return self.bounded(f"aReady{sl}", u)

        def next_row():
            nonlocal slot, use
            self.commits.append(f"aEmpty{slot}")
            slot += 1
            if slot == NS:
                slot, use = 0, use + 1

        for _ in range(units):
            left = 0
            for fc in range(nFC):
                for ky in range(KY):
                    if left == 0:
                        left = self.per_chain
                        if cc >= 2 and not (yield from self.bounded(f"chainEmpty{cc & 1}", (cc >> 1) - 1)):
                            ok = False
                            break
                    for j in range(0 if ky == 0 else R - 1, R):
                        ok = ok and (yield from row(j))
                    if not ok:
                        break
                    for _ in range(KX):
                        if not seen and not (yield from self.bounded(f"bFull{d}", tile)):
                            ok = False
                            break
                        dn, tn = (0, tile + 1) if d + 1 == NB else (d + 1, tile)
                        yield "step"  # half of the tile's MMAs
                        seen = self.carry and self.test(f"bFull{dn}", tn)
                        yield "step"
                        self.commits.append(f"bEmpty{d}")
                        d, tile = dn, tn
                    if not ok:
                        break
                    next_row()
                    left -= 1
                    if left == 0 or (ky + 1 == KY and fc + 1 == nFC):
                        left = 0
                        self.commits.append(f"chainFull{cc & 1}")
                        cc += 1
                if not ok:
                    break
                for _ in range(R - 1):
                    next_row()
            if not ok:
                break
        self.commits.append("done")
        yield from self.wait("done", 0)
        self.left += 1

    def split(self):
        R, NS, NR, NB, KX, KY, nFC, units = self.p
        for c in range(units * nFC * (R + KY - 1)):
            if not (yield from self.bounded(f"rawFull{c % NR}", c // NR)):
                break
            if c >= NS and not (yield from self.bounded(f"aEmpty{c % NS}", c // NS - 1)):
                break
            yield "step"
            self.arrive(f"aReady{c % NS}")
            self.arrive(f"rawEmpty{c % NR}")
        self.left += 1

    def epilogue(self):
        *_, units = self.p
        for cc in range(units * self.chains):
            if not (yield from self.bounded(f"chainFull{cc & 1}", cc >> 1)):
                break
            yield "step"
            self.arrive(f"chainEmpty{cc & 1}")
        self.left += 1

    def run(self):
        roles = {"tma": self.producer(), "mma": self.mma()}
        for w in range(4):
            roles[f"split{w}"], roles[f"epi{w}"] = self.split(), self.epilogue()
        self.play(roles)
        return not self.abort


@pytest.mark.parametrize("R", [1, 2, 3, 4])
def test_every_role_ends_on_a_phase_boundary(R):
    for NS in (R + 1, R + 2):
        for NR in (1, 2):
            for NB in (1, 2, 3, 8):
                for KX, KY in ((1, 1), (3, 3), (7, 7), (9, 5)):
                    for nFC, units in ((1, 0), (1, 1), (3, 1), (1, 3)):
                        c = Conv(R, NS, NR, NB, KX, KY, nFC, units, seed=R + NS + NB + KX + units)
                        what = (R, NS, NR, NB, KX, KY, nFC, units)
                        assert c.run() and c.limits == 0, what
                        assert not c.aliased and not any(c.pending.values()) and not c.in_flight() and not c.commits, what


SMALL = [(2, 3, 2, 3, 3, 3, 1, 1), (1, 2, 1, 2, 3, 1, 2, 1), (2, 4, 2, 8, 1, 3, 1, 2), (4, 5, 2, 2, 3, 3, 1, 1)]


def keys(p):
    R, _, _, _, KX, KY, nFC, units = p
    return [("a", i) for i in range(units * nFC * (R + KY - 1))] + [("b", i) for i in range(units * nFC * KY * KX)]


@pytest.mark.parametrize("p", SMALL)
def test_no_copy_in_flight_at_exit(p):
    for late in keys(p):
        for after in (1, 2):
            c = Conv(*p, seed=3, late={late}, after=after)
            assert not c.run() and c.limits <= 2 * len(keys(p))
            assert c.in_flight() <= c.given_up_landing, (late, after)


def test_a_drain_by_the_producer_alone_is_caught():
    """The last weight tile late: the producer has long issued it and gone on when the MMA warp gives up."""
    for p in SMALL:
        c = Conv(*p, seed=1, late={keys(p)[-1]}, after=2, drain_all=False)
        assert not c.run() and c.in_flight() > c.given_up_landing
