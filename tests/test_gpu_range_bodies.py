"""The range kernel's bodies of 32 and of 24 warps per block, each fixed by a variant of its own, against
the oracle: values of two, three and four words, both signs, with blocks of few and of many rows."""
import os

import pytest

pytestmark = pytest.mark.gpu

NT = max(1, min(32, os.cpu_count() or 1))

RANGES = [
    # (offset, size, k)
    ((1 << 16) - 700, 40000, 8),               # seeds below and above 2^16
    ((1 << 40) + 12345, 1 << 21, 24),          # two words
    ((1 << 60) + (3 << 20) - 5, 1 << 21, 16),  # three words, runs of 32 rows
    ((1 << 90) + 777, 1 << 20, 20),            # four words
]


@pytest.mark.parametrize("negative", [False, True])
@pytest.mark.parametrize("variant", [6, 7])
@pytest.mark.parametrize("case", RANGES, ids=lambda c: f"o{c[0]:x}-s{c[1]}-k{c[2]}")
def test_body_matches_oracle(verifier, case, variant, negative):
    import collatz_b200 as cb
    from oracle import oracle as O
    off, size, k = case
    v = verifier(26)
    v.set_variant(cb.MODE_RANGE, variant)
    v.set_variant(cb.MODE_RANGE64, variant)
    try:
        g = v.verify_range(off, size, k, negative=negative)
    finally:
        v.set_variant(cb.MODE_RANGE, 0)
        v.set_variant(cb.MODE_RANGE64, 0)
    o = O.range_verify(off, size, k, True, method=1, nthreads=NT, negative=negative)
    assert g.errors == 0
    assert (g.seeds_checked, g.failures) == (o.seeds, o.failures)
    assert (g.max_stopping_time, g.max_stopping_time_seed) == (o.max_st, o.max_st_seed)
    assert (g.max_excursion, g.max_excursion_seed) == (o.max_exc, o.max_exc_seed)
