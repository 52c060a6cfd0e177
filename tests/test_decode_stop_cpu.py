"""How a half of a decode CTA (csrc/decode.cu) ends when a wait runs out, on a model of its roles: a producer that
fills a ring, eight warps that take every step and meet at a barrier without a limit once per unit.  Random schedules;
a warp left at the barrier, or a copy still under way when all roles have left, is an error."""
import random

import pytest

WARPS, UNIT = 4, 3   # fewer than the kernel's, the rules do not depend on it


class Half:
    """One half; every method call is one atomic step of one role.  A phase of a ring slot's barriers is counted, not
    its parity alone, except where the kernel compares a ring position."""

    def __init__(self, ring, steps, fail_at, rule, rng):
        self.ring, self.steps, self.fail_at, self.rule, self.rng = ring, steps, fail_at, rule, rng
        self.issued, self.landed, self.end_mark, self.stop_at, self.abort = 0, 0, None, None, False
        self.taken = [0] * WARPS             # steps consumed by each warp
        self.at_barrier = [0] * WARPS        # meetings each warp has come to
        self.left = [False] * WARPS
        self.producer_left = False

    def position(self, step):
        return step % self.ring, step // self.ring % 2

    def producer(self):
        if self.producer_left:
            return False
        slot_free = min(self.taken) > self.issued - self.ring
        gives_up = self.issued >= self.fail_at or (self.abort and self.rng.random() < 0.5)   # the flag is polled on slow paths
        if gives_up or (self.issued == self.steps and slot_free):
            if gives_up:
                self.abort, self.stop_at = True, self.position(self.issued)
            else:
                self.end_mark = self.issued
            self.producer_left = True
            return True
        if self.issued < self.steps and slot_free:
            self.issued += 1
            return True
        return False

    def copy_lands(self):
        if self.landed < self.issued:
            self.landed += 1
            return True
        return False

    def warp(self, w):
        if self.left[w]:
            return False
        n = self.taken[w]
        if n and n % UNIT == 0 and self.at_barrier[w] < n // UNIT:
            self.at_barrier[w] += 1          # stores its sums and comes to the meeting
            return True
        if self.at_barrier[w] and min(self.at_barrier) < self.at_barrier[w]:
            return False                     # stands there, without a limit
        if self.landed > n:
            self.taken[w] += 1
            return True
        if self.end_mark == n:
            self.left[w] = True
            return True
        gives_up = self.stop_at == self.position(n) if self.rule == "position" else self.abort and self.rng.random() < 0.5
        if gives_up:
            self.left[w] = True
            self.abort = True
            return True
        return False

    def run(self, other_half_fails):
        """True if every role leaves."""
        for _ in range(4000):
            if all(self.left) and self.producer_left and self.landed == self.issued:
                return True
            if other_half_fails and self.rng.random() < 0.02:
                self.abort = True
            roles = [self.producer, self.copy_lands] + [lambda w=w: self.warp(w) for w in range(WARPS)]
            self.rng.choice(roles)()
        return False


def ended(rule, trials=1500):
    rng = random.Random(7)
    good = 0
    for _ in range(trials):
        steps = UNIT * rng.randrange(0, 8)
        half = Half(rng.choice((4, 5)), steps, rng.choice((steps + 1, rng.randrange(0, steps + 1))), rule, rng)
        good += half.run(other_half_fails=rng.random() < 0.5)
        assert all(t <= half.issued for t in half.taken)
    return good / trials


def test_every_warp_of_a_half_leaves():
    assert ended("position") == 1.0


def test_the_model_sees_a_warp_left_behind():
    """Each warp looking at the flag for itself, as it should not be."""
    assert ended("flag") < 0.99
