"""Pair batches of every form that the entry point accepts, on the table-driven kernel (variant 4) and on
the four-limb kernel (variant 3): the same hash, counts, errors, overflow seeds and maxima.  Seeds below 3
are reported whatever their numbers' width; bases and numbers of up to 96 and 128 bits, factors 3^f
beyond 2^96, and small checkpoint caps are accepted as well."""
import random

import pytest

pytestmark = pytest.mark.gpu

ERR_ITER_CAP, ERR_SEED_SMALL = 0x2, 0x8


def _key(r):
    return (r.hash, r.seeds_checked, r.errors, r.n_overflow, sorted(r.overflow), r.max_excursion,
            r.max_excursion_seed, r.max_stopping_time, r.max_stopping_time_seed)


def _both(v, bigindex, pairs):
    out = []
    try:
        for variant in (4, 3):
            v.set_variant(0, variant)
            out.append(v.launchkernel(bigindex, pairs, check=False))
    finally:
        v.set_variant(0, 4)
    assert _key(out[0]) == _key(out[1])
    return out[0]


@pytest.mark.parametrize("base", [0, 1, 2])
@pytest.mark.parametrize("bits,bigindex", [(20, 16), (96, 16), (100, 16), (127, 16), (40, 60)])
def test_seeds_below_three_are_reported(verifier, base, bits, bigindex):
    # one of the bases is kept by the mod-9 sieve only; 3^f of bigindex 60 is beyond 2^96
    pairs = [(base, (1 << bits) + 7)]
    r = _both(verifier(26), bigindex, pairs)
    assert r.errors == (ERR_SEED_SMALL if base < 2 else 0)


@pytest.mark.parametrize("n", [16, 26, 36, 40, 45, 52])
@pytest.mark.parametrize("cap", [0, 1, 3, 150])
def test_random_pairs(n, cap):
    import collatz_b200 as cb
    rng = random.Random(n * 1000 + cap)
    with cb.Verifier(n, iter_cap=cap) as v:
        for bigindex in (0, 8, 15, 16, 50):
            for kind in range(3):
                pairs = [(rng.getrandbits(n - 10) if kind == 0 else rng.randrange(4) if kind == 1
                          else rng.getrandbits(rng.randrange(1, 97)), rng.getrandbits(rng.randrange(1, 129)))
                         for _ in range(40)]
                r = _both(v, bigindex, pairs)
                assert r.errors & ~(ERR_ITER_CAP | ERR_SEED_SMALL) == 0
