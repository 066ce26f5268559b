"""A model of what a CTA of k_router_near (csrc/s14_router.cu) does when a wait of one of its threads runs out, run on the CPU: no wait is made to
run out on a GPU.

The CTA's threads load the four stages of a ring, meet at a barrier, one of them queues the step's multiplications, and each waits by itself for
step c - 1 before it loads step c + 3 into that step's stage.  Properties: no thread loads into a stage that queued multiplications still read;
logits that are stored as numbers are those of undisturbed and complete multiplications; tensor memory goes back behind them."""
import random

STAGES, LIMIT = 4, 1000.0   # a wait's limit, in units of a try's length


def run(rng, together, steps):
    """Returns (loads into stages that are being read, threads that store numbers they should not, tensor memory freed too early).  together:
    the threads agree on what they saw at every barrier, stop, and wait for what is queued; else each goes on by itself."""
    n, now = 6, 0.0
    late = rng.randrange(0, 2 * steps)             # the step, if any, that takes longer than a wait
    ok, at, done, torn = [True] * n, [0.0] * n, [], 0
    for c in range(steps):
        now = max(at)                              # the barrier in front of the step's multiplications
        if together:
            ok = [all(ok)] * n
            if not ok[0]:
                break
        done.append(max(now, done[-1] if done else 0.0) + (rng.uniform(0.9, 1.5) * LIMIT if c == late else rng.uniform(0.5, 2.0)))
        at = [now] * n
        if c >= 1 and c + STAGES - 1 < steps:
            for i in range(n):
                start = now + rng.uniform(0.0, 0.2) * LIMIT
                at[i] = min(max(start, done[c - 1]), start + LIMIT)
                if at[i] < done[c - 1]:
                    ok[i] = False
                if ok[i] or not together:
                    torn += at[i] < done[c - 1]    # its load into stage (c - 1) % 4
    last = done[-1]
    for i in range(n):
        if ok[i] or not together:
            start = at[i]
            at[i] = min(max(start, last), start + LIMIT)
            ok[i] = ok[i] and at[i] >= last
    now = max(at)
    if together:
        ok = [all(ok)] * n
        if not ok[0]:
            now = min(max(now, last), now + LIMIT)
    return torn, sum(o and (torn > 0 or now < last) for o in ok), now < last


def outcomes(together):
    rng = random.Random(5)
    runs = [run(rng, together, rng.randrange(1, 9)) for _ in range(20_000)]
    return [sum(r[k] > 0 for r in runs) for k in range(3)]


def test_a_cta_that_gave_up_disturbs_nothing_and_claims_nothing():
    assert outcomes(together=True) == [0, 0, 0]


def test_threads_that_go_on_by_themselves_do():
    assert min(outcomes(together=False)) > 0
