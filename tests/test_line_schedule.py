"""CPU model of the line-scan sweeps' hand-overs (tbl_line.cu): the rings' slots,
the mbarrier phases, the carry mailboxes, the exchange between CTAs and the tickets,
under random schedules.

Agents are the kernel's: the feeder's bulk copies (which land whenever they like),
the couriers, and the sweeping warps, each stepping between the points where it
touches something shared.  Checked: every row meets its own operands, its plane
below and its carry; no slot is overwritten before it has been read; a wait that
tests a parity never mistakes one phase for another; nothing waits for ever, with
as few as one CTA resident; the exchange words and the tickets end as they began."""
import os
import random
import re

import pytest

SRC = open(os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "turbulentbl_gb300", "csrc",
                        "tbl_line.cu")).read()
XR = int(re.search(r"LINE_XR = (\d+);", SRC).group(1))
H = XR // 2


class Barrier:
    """An mbarrier of one arrival and counted transactions."""

    def __init__(self):
        self.phase, self.pending, self.tx = 0, 1, 0

    def _turn(self):
        if self.pending == 0 and self.tx == 0:
            self.phase, self.pending = self.phase + 1, 1

    def arrive(self, expect=0):
        assert self.pending == 1, "a second arrival in one phase"
        self.tx += expect
        self.pending = 0
        self._turn()

    def land(self):
        self.tx -= 1
        self._turn()

    def test(self, n):
        """Whether phase n is over, as its parity tells."""
        over = (self.phase & 1) != (n & 1)
        assert over == (self.phase > n) and self.phase <= n + 1, "a parity of another phase"
        return over


class Warp:
    """Ring, barriers and mailbox of one sweeping warp."""

    def __init__(self):
        self.op, self.below = [None] * XR, [None] * XR
        self.full = [Barrier() for _ in range(XR)]
        self.empty, self.opfull = [Barrier(), Barrier()], [Barrier(), Barrier()]
        self.mail = {}
        self.read = -1  # last row whose slot has been read


class Model:
    def __init__(self, K, KP, S, nrow, resident, seed):
        self.K, self.KP, self.S, self.nrow = K, KP, S, nrow
        self.rng = random.Random(seed)
        self.xch, self.copies, self.done = {}, [], set()
        self.waiting = list(range((K + KP - 1) // KP))  # tickets: lowest planes first
        self.running = []  # (CTA, its agents)
        self.resident = resident

    def start(self):
        while self.waiting and len(self.running) < self.resident:
            kg = self.waiting.pop(0)
            live = [(kp, s) for kp in range(self.KP) if kg * self.KP + kp < self.K for s in range(self.S)]
            warps = {q: Warp() for q in live}
            agents = [self.feed(warps[q]) for q in live] + [self.sweep(kg, q, warps) for q in live]
            if kg > 0:
                agents += [self.courier(kg, s, warps[0, s]) for s in range(self.S)]
            self.running.append([kg, agents])

    # ---- agents: generators that yield False while they wait
    def feed(self, w):
        nh = (self.nrow + H - 1) // H
        for m in range(nh):
            while m >= 2 and not w.empty[m & 1].test(m // 2 - 1):
                yield False
            n = min(H, self.nrow - m * H)
            w.opfull[m & 1].arrive(n)
            for r in range(m * H, m * H + n):
                self.copies.append((w, r))
                yield True
        for m in range(max(0, nh - 2), nh):
            while not w.opfull[m & 1].test(m // 2):
                yield False

    def land(self):
        w, r = self.copies.pop(self.rng.randrange(len(self.copies)))
        assert w.op[r % XR] is None or w.op[r % XR] <= w.read, "operands not read yet"
        w.op[r % XR] = r
        w.opfull[r % XR // H].land()

    def put_below(self, w, plane, r):
        old = w.below[r % XR]
        assert old is None or old[1] <= w.read, "a row of the plane below not read yet"
        w.below[r % XR] = (plane, r)
        w.full[r % XR].arrive()

    def courier(self, kg, s, w):
        for r in range(self.nrow):
            while r % H == 0 and r >= XR and not w.empty[r % XR // H].test(r // XR - 1):
                yield False
            while self.xch.get((kg - 1, s, r)) is None:
                yield False
            self.put_below(w, self.xch.pop((kg - 1, s, r)), r)
            yield True

    def sweep(self, kg, q, warps):
        kp, s = q
        plane, w = kg * self.KP + kp, warps[q]
        above = warps.get((kp + 1, s))

        def there(r):
            return w.full[r % XR] if plane > 0 else w.opfull[r % XR // H]

        def ready(r):
            ok = there(r).test(r // XR)
            return (r % H != 0 or w.opfull[r % XR // H].test(r // XR)) and ok

        def take(r):
            assert w.op[r % XR] == r, "another row's operands"
            assert plane == 0 or w.below[r % XR] == (plane - 1, r), "another row of the plane below"
            w.read = r

        while not ready(0):
            yield False
        take(0)
        for r in range(self.nrow):
            more = r + 1 < self.nrow
            early = more and ready(r + 1)
            if early:
                take(r + 1)
            yield True
            while s > 0 and r not in warps[kp, s - 1].mail:
                yield False
            w.mail[r] = True
            yield True
            if plane + 1 < self.K:
                if kp < self.KP - 1:
                    while r % H == 0 and r >= XR and not above.empty[r % XR // H].test(r // XR - 1):
                        yield False
                    self.put_below(above, plane, r)
                else:
                    assert (kg, s, r) not in self.xch, "a row not taken yet"
                    self.xch[kg, s, r] = plane
                yield True
            self.done.add((plane, s, r))
            if more and not early:
                while not ready(r + 1):
                    yield False
                take(r + 1)
            if more and (r + 1) % H == H - 1 and r + 1 + H + 1 < self.nrow:
                w.empty[(r + 1) % XR // H].arrive()

    # ---- schedule
    def run(self):
        idle = 0
        while True:
            self.start()
            if not self.running:
                break
            moved = False
            if self.copies and self.rng.random() < 0.3:
                self.land()
                moved = True
            cta = self.rng.choice(self.running)
            a = self.rng.choice(cta[1])
            try:
                moved = next(a) or moved
            except StopIteration:
                cta[1].remove(a)
                moved = True
                if not cta[1]:
                    self.running.remove(cta)
            idle = 0 if moved else idle + 1
            if idle > 2000:
                assert self.copies, "everything waits"
                self.land()
                idle = 0
        assert not self.copies and not self.xch
        assert len(self.done) == self.K * self.S * self.nrow


@pytest.mark.parametrize("resident", [1, 3])
@pytest.mark.parametrize("K,KP,S", [(1, 1, 1), (5, 1, 1), (4, 2, 1), (7, 3, 2), (3, 4, 3), (6, 1, 4), (9, 4, 1)])
@pytest.mark.parametrize("nrow", [4, 5, 7, 8, 9, 12, 13, 16, 17, 32])
def test_every_schedule_completes(nrow, K, KP, S, resident):
    for seed in range(6):
        Model(K, KP, S, nrow, resident, seed).run()
