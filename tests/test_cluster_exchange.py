"""Host model of the two-CTA exchange of blind_rotate_latency.cu: each step a CTA expects the other's bytes on the
step's receive barrier (one of two, by parity), sends its own spectrum, which lands there at any later time, and
waits; a wait that runs out, or a raised abort flag, ends the CTA's loop at the end of a later step.  After the cluster
barrier a CTA whose flag is up waits for every spectrum that it was sent before it exits.

The model runs both CTAs at random speeds, lets waits run out and flags rise at random, and checks the barrier's rules
(one arrival a phase, none while a phase's bytes are missing), that every run ends and that nothing lands in a CTA
that has exited."""
import numpy as np
import pytest

BYTES = 3


class Barrier:
    """mbarrier with one expected arrival: phase k completes once it was armed and its bytes have landed."""

    def __init__(self):
        self.phase, self.armed, self.tx = 0, False, 0

    def settle(self):
        if self.armed and self.tx == 0:
            self.phase, self.armed = self.phase + 1, False

    def expect(self):
        assert not self.armed, "arrival in a phase that has had its one"
        self.armed, self.tx = True, self.tx + BYTES
        self.settle()

    def land(self):
        self.tx -= BYTES
        self.settle()

    def done(self, parity):  # what a parity wait sees
        return (self.phase & 1) != parity


class Cluster:
    def __init__(self, nsteps, rng, quit_rate, drain):
        self.rng, self.nsteps, self.quit_rate, self.drain = rng, nsteps, quit_rate, drain
        self.bars = [[Barrier(), Barrier()] for _ in range(2)]
        self.flag, self.steps, self.at_barrier, self.exited = [False] * 2, [0, 0], [False] * 2, [False] * 2
        self.flying = []  # [time to land, CTA, barrier]

    def cta(self, r):
        steps, stop = 0, False
        while steps < self.nsteps and not stop:
            stop = self.flag[r]
            self.bars[r][steps & 1].expect()
            yield
            slow = self.rng.random() < .2
            self.flying.append([int(self.rng.integers(1, 60 if slow else 4)), 1 - r, steps & 1])
            if self.rng.random() < self.quit_rate:  # a wait for the key ran out, in this warp or the producer's
                self.flag[r] = True
            yield
            while not self.flag[r] and not self.bars[r][steps & 1].done(steps >> 1 & 1):
                if self.rng.random() < self.quit_rate or self.flag[1 - r] and self.at_barrier[1 - r]:
                    self.flag[r] = True  # the wait ran out
                yield
            steps += 1
            yield
        self.steps[r] = steps
        self.at_barrier[r] = True
        while not all(self.at_barrier):
            yield
        if self.flag[r] and self.drain:
            sent = self.steps[1 - r]
            assert abs(sent - steps) <= 2
            for s in range(max(0, min(steps, sent) - 2), sent):
                if s >= steps:
                    self.bars[r][s & 1].expect()
                while not self.bars[r][s & 1].done(s >> 1 & 1):
                    yield
        self.exited[r] = True

    def run(self):
        live = {r: self.cta(r) for r in range(2)}
        for _ in range(200000):
            for f in self.flying:
                f[0] -= 1
            landed = [f for f in self.flying if f[0] <= 0]
            self.flying = [f for f in self.flying if f[0] > 0]
            for _, r, p in landed:
                assert not self.exited[r], "a spectrum landed in a CTA that has exited"
                self.bars[r][p].land()
            for r in list(live):
                if self.rng.random() < .7:
                    try:
                        next(live[r])
                    except StopIteration:
                        del live[r]
            if not live and not self.flying:
                return
        raise AssertionError("deadlock")


@pytest.mark.parametrize("nsteps", [1, 2, 3, 4, 9])
@pytest.mark.parametrize("quit_rate", [0.0, 0.01, 0.1, 0.5])
def test_nothing_lands_after_the_exit(nsteps, quit_rate):
    rng = np.random.default_rng(1000 * nsteps + int(100 * quit_rate))
    for _ in range(400):
        Cluster(nsteps, rng, quit_rate, drain=True).run()


@pytest.mark.parametrize("nsteps", [1, 9])
def test_model_detects_an_exit_right_after_the_cluster_barrier(nsteps):
    # the barrier alone, which does not order the asynchronous stores
    rng = np.random.default_rng(nsteps)
    with pytest.raises(AssertionError, match="exited"):
        for _ in range(400):
            Cluster(nsteps, rng, 0.1, drain=False).run()
