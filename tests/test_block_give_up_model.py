"""Models of what a pair of CTAs of the block kernels (csrc/s14_moe_pair.cu) does when a wait of one of its roles runs out,
run on the CPU: no wait is made to run out on a GPU, because the stages' waits have no limit that a test could shorten.

Leaving.  The first CTA's issuing warp has queued stages of tensor operations that run in order; they read both CTAs'
shared memory, write both CTAs' tensor memory and arrive at barriers of both.  A role that gives up raises its CTA's flag, the
CTA's other roles follow at their next wait, and the CTA walks to its end: the issuing warp commits a last arrival (`fin`)
behind all that is queued, both CTAs meet at the cluster barrier, free their tensor memory and leave.  Property: when a
CTA frees and leaves, every queued operation is complete and every arrival at that CTA's barriers has come."""
import random

import pytest

LIMIT = 1000.0   # a wait's limit, in units of a try's length


def leave(rng, drain):
    """One random ending; returns (times the two CTAs leave, time the operations end, time the last arrival reaches CTA 1)."""
    queued, stage, hop = rng.randrange(0, 13), rng.uniform(0.1, 0.5), rng.uniform(0.0, 2.0)
    # one CTA's role gives up; the other one's notices when a wait on the first runs out, up to a limit later
    first, other = rng.uniform(0.0, 10.0), rng.uniform(0.0, 1.0) * LIMIT
    end = [first, first + other] if rng.random() < 0.5 else [first + other, first]
    # (stages that were there before the first CTA's issuing warp stopped)
    ops_done = end[0] + queued * stage
    fin = ops_done                          # in the first CTA; in the second a hop later
    if drain:                               # the first waits for it whatever the flag says, the second behind the cluster barrier
        at_barrier = [min(max(end[0], fin), end[0] + LIMIT), end[1]]
        met = max(at_barrier)
        return (met, min(max(met, fin + hop), met + LIMIT)), ops_done, fin + hop
    at_barrier = [min(max(e, f), e + 1.0) for e, f in zip(end, (fin, fin + hop))]   # one try once the flag is up
    met = max(at_barrier)
    return (met, met), ops_done, fin + hop


def sound(ending):
    (left0, left1), ops_done, arrived1 = ending
    return ops_done <= min(left0, left1) and arrived1 <= left1


def test_a_pair_that_gave_up_leaves_behind_its_tensor_work():
    rng = random.Random(7)
    assert all(sound(leave(rng, drain=True)) for _ in range(20_000))


def test_a_wait_that_ends_with_the_flag_would_leave_work_in_flight():
    rng = random.Random(7)
    assert not all(sound(leave(rng, drain=False)) for _ in range(20_000))


# ---- publishing ----
# A rank's call is two contraction kernels, every CTA of which may give up; a CTA that did has not stored its rows (down) or the
# hidden values they are made of (up).  The CTAs of the second kernel count themselves in, in any order, and the last one publishes.


def publish(rng, n_ctas, call, up_gave_up, down_gave_up, by_word, word):
    """The number the last CTA publishes.  by_word: it reads the call's word, which every CTA that gave up has set before
    it counted itself in; else its own flag."""
    word = 0 if by_word else word           # the call's grouping sets it anew
    if up_gave_up:
        word = 1
    order = rng.sample(range(n_ctas), n_ctas)
    for cta in order:
        word |= cta in down_gave_up
    failed = word if by_word else order[-1] in down_gave_up
    return (0 if failed else call), word


@pytest.mark.parametrize("by_word", [True, False])
def test_a_call_with_a_cta_that_gave_up_is_not_published(by_word):
    rng = random.Random(11)
    wrong, word, n = 0, 0, 8
    for call in range(1, 2001):
        up = {c for c in range(n) if rng.random() < 0.03}
        down = {c for c in range(n) if rng.random() < 0.03}
        # an up kernel that gave up leaves hidden values of an earlier call, which the down kernel works on
        number, word = publish(rng, n, call, bool(up), down, by_word, word)
        wrong += number != (0 if up or down else call)
    assert (wrong == 0) == by_word
