"""A batch of tens of thousands of small requests: more candidates than a launch's list holds (2^16: the
rest take their records' locks in the kernel), settled for the requests of a warp's lanes side by
side.  Every request gets the oracle's result for it alone, in a batch and in a plan."""
import random

import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,top,k,negative", [(40000, 300, 16, False), (5000, 600, 12, True), (33, 40, 24, False)])
def test_many_small_requests(verifier, n, top, k, negative):
    from oracle import oracle as O
    rng = random.Random(n)
    reqs = [(rng.randrange(1 << 40, 1 << 62), rng.randint(1, top), k, True, negative) for _ in range(n)]
    reqs[n // 2:n // 2 + 8] = reqs[:8]  # some twice
    v = verifier(26)
    got = v.verify_batch(reqs)
    plan = v.plan(reqs)
    try:
        plan.launch()
        again = plan.results()
    finally:
        plan.close()
    key = lambda r: (r.seeds_checked, r.failures, r.max_stopping_time, r.max_stopping_time_seed, r.max_excursion,  # noqa: E731
                     r.max_excursion_seed, r.errors)
    offers = 0
    for q, a, b in zip(reqs, got, again):
        o = O.range_verify(*q[:4], method=1, nthreads=1, negative=negative)
        assert key(a) == key(b) == (o.seeds, o.failures, o.max_st, o.max_st_seed, o.max_exc, o.max_exc_seed, 0), q
        offers += 2 * (o.seeds > 0)
    assert n < 40000 or offers > 1 << 16
