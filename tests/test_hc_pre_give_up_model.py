"""A model of how the CTAs of a cluster of k_hc_pre (csrc/s14_glue.cu) leave when the sums of some have not come to others in a wait's length, run on
the CPU: no wait is made to run out on a GPU.

Every CTA stores its sums into all of them, each store on its way for a while, waits (bounded) for all that it is to get, and leaves.  Property:
no store arrives in a CTA that has left."""
import random

CTAS, LIMIT = 16, 1000.0   # a wait's limit, in units of a try's length


def late_arrivals(rng, stays):
    """Stores that arrive in CTAs that have left.  stays: a CTA that gave up waits for the others to leave or to give up, and then for what is on
    its way; else it leaves."""
    start = [rng.uniform(0.0, 5.0) for _ in range(CTAS)]
    if rng.random() < 0.7:                         # one of them is far behind
        start[rng.randrange(CTAS)] += rng.uniform(0.5, 3.0) * LIMIT
    arrive = [[start[f] + rng.uniform(0.5, 3.0) for _ in range(CTAS)] for f in range(CTAS)]   # [from][to]
    all_come = [max(arrive[f][to] for f in range(CTAS)) for to in range(CTAS)]
    seen = [min(max(start[to], all_come[to]), start[to] + LIMIT) for to in range(CTAS)]
    gave_up = [seen[to] < all_come[to] for to in range(CTAS)]
    leaves = list(seen)
    if stays:
        met = max(seen)                            # everyone has left or is at the barrier
        leaves = [min(max(met, all_come[to]), met + LIMIT) if gave_up[to] else seen[to] for to in range(CTAS)]
    return sum(arrive[f][to] > leaves[to] for f in range(CTAS) for to in range(CTAS))


def test_no_sum_arrives_in_a_cta_that_has_left():
    rng = random.Random(3)
    assert sum(late_arrivals(rng, stays=True) for _ in range(3000)) == 0


def test_a_cta_that_gave_up_and_left_would_be_written_to():
    rng = random.Random(3)
    assert sum(late_arrivals(rng, stays=False) for _ in range(3000)) > 0
