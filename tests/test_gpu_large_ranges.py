"""Ranges of 2^30 to 2^34 seeds, of every width and both signs, against the CPU oracle's results
(tests/golden/large_ranges.json, made by tests/golden/make_large_range_golden.py): on such sizes the
kernel's windows decide nearly every seed by its bounds alone.  With the default and with each fixed body;
ranges that fit two words with three as well."""
import pytest

from conftest import load_golden

pytestmark = pytest.mark.gpu

FIXTURES = load_golden("large_ranges.json")


@pytest.mark.parametrize("variant", [0, 6, 7])
@pytest.mark.parametrize("i", range(len(FIXTURES)))
def test_large_range_matches_oracle(verifier, i, variant):
    import collatz_b200 as cb
    g = FIXTURES[i]
    off, size = int(g["offset"]), int(g["size"])
    want = (g["seeds"], g["failures"], g["max_stopping_time"], int(g["max_stopping_time_seed"]),
            int(g["max_excursion"]), int(g["max_excursion_seed"]), 0)
    v = verifier(26)
    try:
        v.set_variant(cb.MODE_RANGE, variant)
        v.set_variant(cb.MODE_RANGE64, variant)
        for bits in ([48, 0] if (off + size - 1).bit_length() <= 48 else [48]):
            v.set_variant(cb.MODE_RANGE64_BITS, bits)
            r = v.verify_range(off, size, g["k"], g["mod9"], negative=g["negative"])
            assert (r.seeds_checked, r.failures, r.max_stopping_time, r.max_stopping_time_seed, r.max_excursion,
                    r.max_excursion_seed, r.errors) == want, bits
    finally:
        v.set_variant(cb.MODE_RANGE, 0)
        v.set_variant(cb.MODE_RANGE64, 0)
        v.set_variant(cb.MODE_RANGE64_BITS, cb.RANGE64_BITS_DEFAULT)
