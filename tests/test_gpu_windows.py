"""The table-driven steps on the GPU against the oracle, at the sizes where they can go
wrong: seeds around 2^16 (windows from there on), the widths at which a value gets
another word, runs longer than a run's limit, partial rows, both signs, with and
without the mod-9 sieve; and pair batches whose values lie around the limits of the
three words kept and of the exact path."""
import os

import pytest

pytestmark = pytest.mark.gpu

NT = max(1, min(32, os.cpu_count() or 1))

RANGES = [
    # (offset, size, k)
    ((1 << 16) - 700, 1500, 8),           # seeds below and above 2^16, partial blocks
    (1 << 20, 3 << 20, 8),                # 12 288 blocks of few residues: runs at their limit
    ((1 << 40) + 9, 1, 16),               # one seed, or none
    ((1 << 40) + (7 << 16), 1 << 16, 16), # one whole block
    ((1 << 48) - (1 << 17) + 5, 1 << 18, 16),   # 48 and 49 bits: two and three words
    ((1 << 80) - (1 << 17) + 5, 1 << 18, 16),   # 80 and 81 bits: three and four words
]


@pytest.mark.parametrize("negative", [False, True])
@pytest.mark.parametrize("mod9", [True, False])
@pytest.mark.parametrize("case", RANGES, ids=lambda c: f"o{c[0]:x}-s{c[1]}-k{c[2]}")
def test_range_windows_match_oracle(verifier, case, mod9, negative):
    from oracle import oracle as O
    off, size, k = case
    g = verifier(26).verify_range(off, size, k, mod9, negative=negative)
    o = O.range_verify(off, size, k, mod9, method=1, nthreads=NT, negative=negative)
    assert g.errors == 0
    assert (g.seeds_checked, g.failures) == (o.seeds, o.failures)
    assert (g.max_stopping_time, g.max_stopping_time_seed) == (o.max_st, o.max_st_seed)
    assert (g.max_excursion, g.max_excursion_seed) == (o.max_exc, o.max_exc_seed)


@pytest.mark.parametrize("bits", [16, 48, 64, 71, 72, 80, 96])
@pytest.mark.parametrize("n", [26, 45])
def test_pair_look_ups_match_oracle(verifier, oracle_tables, n, bits):
    v, T = verifier(n), oracle_tables(n)
    mask = (1 << (n - 10)) - 1
    pairs = [((0x9E3779B97F4A7C15 * (i + 1)) & mask, (1 << bits) - 12345 + 4097 * i) for i in range(8)]
    pairs += pairs[:1] * 40  # more pairs than a warp's slots
    pairs += [(pairs[1][0], 0)]  # a value of 0 for a = 0
    r = v.launchkernel(3, pairs)
    o = T.pairs_result(3, pairs)
    assert (r.hash, r.seeds_checked, r.errors) == (o.hash, o.seeds, 0)
    assert sorted(r.overflow) == sorted(o.overflow)
    assert (r.max_stopping_time, r.max_stopping_time_seed) == (o.max_st, o.max_st_seed)
    assert (r.max_excursion, r.max_excursion_seed) == (o.max_exc, o.max_exc_seed)
