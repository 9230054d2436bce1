"""Generates tests/golden/large_ranges.json: ranges of 2^30 to 2^34 seeds for every width of the range kernel
and both signs, computed by the CPU oracle (method 1, the reference's search3 loop, collatz_cudav7.cu:684-715)
on all host threads.  The kernel never computes most of these seeds exactly, so that its bounds are
compared with an independent answer here, on the sizes where few seeds still count (about two
minutes on 8 cores).

  python tests/golden/make_large_range_golden.py
"""
from __future__ import annotations

import json
import os
import sys

HERE = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, os.path.dirname(os.path.dirname(HERE)))
from oracle import oracle as O  # noqa: E402

RANGES = [
    # (offset, size, k, mod9, negative)
    ((1 << 40) + 12345, 1 << 34, 24, True, False),        # two words
    ((1 << 48) - (1 << 31), 1 << 32, 24, True, False),    # 48 and 49 bits: three words
    ((1 << 60) + 777, 1 << 31, 16, True, False),          # three words, long runs
    ((1 << 80) - (1 << 31) + 5, 1 << 32, 24, True, False),  # 80 and 81 bits: four words
    ((1 << 90) + 777, 1 << 33, 24, True, False),          # four words
    ((1 << 42) + 99, 1 << 30, 20, False, False),          # no mod-9 sieve
    ((1 << 40) + 12345, 1 << 33, 24, True, True),
    ((1 << 60) + 777, 1 << 31, 20, True, True),
    ((1 << 90) + 777, 1 << 31, 24, True, True),
    (2, 1 << 31, 16, True, True),
]


def main():
    out = []
    for off, size, k, mod9, neg in RANGES:
        r = O.range_verify(off, size, k, mod9, 1, os.cpu_count() or 1, negative=neg)
        out.append({"offset": str(off), "size": str(size), "k": k, "mod9": mod9, "negative": neg, "seeds": r.seeds,
                    "failures": r.failures, "max_stopping_time": r.max_st, "max_stopping_time_seed": str(r.max_st_seed),
                    "max_excursion": str(r.max_exc), "max_excursion_seed": str(r.max_exc_seed)})
        print(out[-1], file=sys.stderr)
    with open(os.path.join(HERE, "large_ranges.json"), "w") as f:
        json.dump(out, f, indent=1)
        f.write("\n")


if __name__ == "__main__":
    main()
