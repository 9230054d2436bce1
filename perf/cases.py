"""The work that performance is measured on: what a user's program has this
framework do, through its public entry points, from one small range request
to the largest configured block.

listed() names the cases, draw(rng) gives more of the same ranges, prepare()
makes what a program has in hand before the call, run() is one pass, work()
the bytes and 32-bit operations a pass cannot do without and exact() what
run() returns, from plain Python integers.

Seeds, offsets and lines are drawn from the state's seed; the sizes within a
mix are drawn from the case's own numbers, so that every state of a case is
the same amount of work.  All outputs are whole numbers.  A program keeps one context (or server) per process with the
sieve tables of the exponents it uses, so contexts and servers are made once
and kept here.
"""
import math
import random

import numpy as np

import collatz_b200 as cb

ROOT_CASE = (3, 2, 2, 9, 1, 0)  # the whole Step-1 tree, as one line of a cases file
_kept = {}


# ----------------------------------------------------------------------------
# cases
# ----------------------------------------------------------------------------

def listed():
    return [
        # one small request, as a client with a few million integers to check sends it: launch latency
        {"name": "range_2p20", "kind": "range", "size": (1 << 20) + 77, "k": 24, "lo": 40, "hi": 64, "align": 1},
        # an ordinary request below 2^48, unaligned and of odd size
        {"name": "range_2p30", "kind": "range", "size": (1 << 30) + 12345, "k": 24, "lo": 40, "hi": 47, "align": 1},
        # the plain verification that also runs on a CPU: 2^32 integers from (nearly) zero, 2^16 sieve
        {"name": "plain_2p32_k16", "kind": "range", "size": 1 << 32, "k": 16, "lo": 0, "hi": 16, "align": 1},
        # the single large block: 2^38 seeds at 2^40, 2^24 sieve
        {"name": "block_2p38", "kind": "range", "size": 1 << 38, "k": 24, "lo": 40, "hi": 44, "align": 1 << 24},
        # the frontier block: 2^40 seeds at 2^60, 2^34 sieve
        {"name": "frontier_2p40", "kind": "range", "size": 1 << 40, "k": 34, "lo": 60, "hi": 61, "align": 1 << 34},
        # the negative integers' variant on an ordinary range
        {"name": "negative_2p32", "kind": "range", "size": (1 << 32) + 3, "k": 24, "lo": 40, "hi": 47, "align": 1,
         "negative": True},
        # the batched configuration with fewer requests: uneven sizes in one launch of a kept plan
        {"name": "plan_512", "kind": "plan", "n": 512, "lo_log2": 20, "hi_log2": 34},
        # many small requests in one call
        {"name": "batch_1000_small", "kind": "batch", "n": 1000, "lo_log2": 16, "hi_log2": 20},
        # one full trajectory query: 65536 seeds of 64 to 256 bits
        {"name": "query_65536", "kind": "query", "n": 65536},
        # one line of a cases file near the root: hundreds of millions of seeds at N = 45
        {"name": "line_n45", "kind": "line", "maxbits": 45, "cut": 10},
        # many small lines, the shape of a large cases file, combined by the driver
        {"name": "lines_n45_2048", "kind": "lines", "maxbits": 45, "cut": 24, "n": 2048},
        # a served burst: range requests and trajectory queries in flight together
        {"name": "served_64", "kind": "served", "n": 64, "lo_log2": 16, "hi_log2": 32},
    ]


def _log2(rng, lo, hi):
    return int(2.0 ** rng.uniform(lo, hi))


def draw(rng):
    kind = rng.choice(["range", "range", "range", "range", "plan", "batch", "query", "line", "lines", "pairs", "served"])
    if kind == "range":
        negative = rng.random() < 0.15
        k = rng.choice([16, 20, 24, 24, 24])
        lo = rng.randrange(k, 63)
        return {"kind": "range", "size": _log2(rng, 16, 34 if negative else 37), "k": k, "lo": lo,
                "hi": rng.randrange(lo + 1, 65), "align": rng.choice([1, 1, 1 << k]), "negative": negative,
                "mod9": rng.random() < 0.9}
    if kind == "plan":
        return {"kind": "plan", "n": _log2(rng, 4, 9), "lo_log2": rng.randrange(18, 24), "hi_log2": rng.randrange(26, 34)}
    if kind == "batch":
        return {"kind": "batch", "n": _log2(rng, 1, 11), "lo_log2": rng.randrange(10, 18), "hi_log2": rng.randrange(19, 23)}
    if kind == "query":
        return {"kind": "query", "n": _log2(rng, 0, 16)}
    if kind == "line":
        return {"kind": "line", "maxbits": rng.choice([36, 40, 42, 45]), "cut": rng.randrange(10, 20)}
    if kind == "lines":
        return {"kind": "lines", "maxbits": rng.choice([36, 40, 45]), "cut": rng.randrange(20, 25), "n": _log2(rng, 3, 11)}
    if kind == "pairs":
        return {"kind": "pairs", "maxbits": rng.choice([36, 42, 45]), "cut": rng.randrange(12, 16), "n": _log2(rng, 4, 14)}
    return {"kind": "served", "n": _log2(rng, 1, 7), "lo_log2": 16, "hi_log2": rng.randrange(24, 33)}


# ----------------------------------------------------------------------------
# what a program keeps
# ----------------------------------------------------------------------------

def _verifier(maxbits=45):
    key = ("verifier", maxbits)
    if key not in _kept:
        _kept[key] = cb.Verifier(maxbits, range_k=24)
    return _kept[key]


def _tables(k, negative):
    """The context with the tables of the 2^k sieve on the device."""
    v = _verifier()
    if ("tables", k, negative) not in _kept:
        v.verify_range(1 << 40, 1 << 16, k, negative=negative)
        _kept[("tables", k, negative)] = True
    return v


def _server():
    if "server" not in _kept:
        s = cb.Server(26, range_k=24)
        for t in (s.submit_range(1 << 50, 1 << 24), s.submit_trajectory_array(_query_seeds(random.Random(1), 1000))):
            s.wait(t)
        _kept["server"] = s
    return _kept["server"]


def _split(maxbits, cut):
    """All lines at sigfig = cut of the whole tree, with at least the root."""
    key = ("split", maxbits, cut)
    if key not in _kept:
        _kept[key] = [cb.case_tuple(c) for c in cb.split_cases(maxbits, ROOT_CASE, cut)]
    return _kept[key]


# ----------------------------------------------------------------------------
# inputs
# ----------------------------------------------------------------------------

def _query_seeds(rng, n):
    """n seeds of 64 to 256 bits (uniform bit lengths) as (n, 8) limbs."""
    g = np.random.default_rng(rng.getrandbits(48))
    bits = g.integers(64, 257, n)
    x = g.integers(0, 1 << 32, size=(n, 8), dtype=np.uint64)
    for j in range(8):
        x[:, j] &= (np.uint64(1) << np.clip(bits - 32 * j, 0, 32).astype(np.uint64)) - np.uint64(1)
    x[np.arange(n), (bits - 1) // 32] |= np.uint64(1) << ((bits - 1) % 32).astype(np.uint64)
    return x.astype(np.uint32)


def _offset(rng, lo, hi, align):
    off = rng.randrange(0 if lo == 0 else 1 << lo, 1 << hi)
    return off - off % align


def _requests(rng, n, lo_log2, hi_log2, align):
    sizes = random.Random(n)
    return [(_offset(rng, 40, 64, align), _log2(sizes, lo_log2, hi_log2), 24, True) for _ in range(n)]


def prepare(case, seed):
    rng = random.Random(seed)
    kind = case["kind"]
    if kind == "range":
        v = _tables(case["k"], case.get("negative", False))
        off = _offset(rng, case["lo"], case["hi"], case["align"])
        return {"kind": kind, "v": v, "args": (off, case["size"], case["k"], case.get("mod9", True)),
                "negative": case.get("negative", False)}
    if kind == "plan":
        v = _tables(24, False)
        return {"kind": kind, "plan": v.plan(_requests(rng, case["n"], case["lo_log2"], case["hi_log2"], 1 << 24))}
    if kind == "batch":
        v = _tables(24, False)
        return {"kind": kind, "v": v, "reqs": _requests(rng, case["n"], case["lo_log2"], case["hi_log2"], 1)}
    if kind == "query":
        return {"kind": kind, "v": _verifier(), "seeds": _query_seeds(rng, case["n"])}
    if kind == "line":
        return {"kind": kind, "v": _verifier(case["maxbits"]), "line": rng.choice(_split(case["maxbits"], case["cut"]))}
    if kind == "lines":
        lines = _split(case["maxbits"], case["cut"])
        n = min(case["n"], len(lines))
        a = rng.randrange(0, len(lines) - n + 1)
        arr = (cb.Case * n)()
        for i in range(n):
            arr[i] = cb.make_case(*lines[a + i])
        return {"kind": kind, "v": _verifier(case["maxbits"]), "lines": arr}
    if kind == "pairs":
        bi, pairs = _pairs(rng, case)
        return {"kind": kind, "v": _verifier(case["maxbits"]), "bigindex": bi, "pairs": cb.pack_pairs(pairs)}
    reqs, mix = [], random.Random(case["n"])
    for _ in range(case["n"]):
        if mix.random() < 0.7:
            reqs.append((_offset(rng, 40, 64, 1), _log2(mix, case["lo_log2"], case["hi_log2"]), 24))
        else:
            reqs.append(_query_seeds(rng, _log2(mix, 0, 16)))
    return {"kind": kind, "server": _server(), "reqs": reqs}


def _pairs(rng, case):
    """Step-1 leaves of one bucket, from as many lines as give n of them."""
    lines = _split(case["maxbits"], case["cut"])
    bi, pairs = None, []
    for line in rng.sample(lines, len(lines)):
        leaves = cb.step1_pairs(case["maxbits"], *line, cap=4 * case["n"])
        if bi is None and leaves:
            b = [x[0] for x in leaves]
            bi = max(set(b), key=b.count)
        pairs += [(x[1], x[2]) for x in leaves if x[0] == bi]
        if len(pairs) >= case["n"]:
            break
    return (0 if bi is None else bi), pairs[:case["n"]]


# ----------------------------------------------------------------------------
# one pass
# ----------------------------------------------------------------------------

def _range_bytes(r):
    return b"".join((r.seeds_checked.to_bytes(8, "little"), r.failures.to_bytes(8, "little"),
                     r.widened.to_bytes(8, "little"), r.max_excursion.to_bytes(32, "little"),
                     r.max_excursion_seed.to_bytes(16, "little"), r.max_stopping_time.to_bytes(8, "little"),
                     r.max_stopping_time_seed.to_bytes(16, "little"), r.errors.to_bytes(4, "little"),
                     (r.status & 0xFFFFFFFF).to_bytes(4, "little")))


def _ranges(results):
    """The results' outputs (all but the device time) as whole numbers, 26 words each."""
    return np.frombuffer(b"".join(map(_range_bytes, results)), dtype=np.int32).reshape(len(results), 26)


def _case(r):
    head = (r.hash, r.launches, r.seeds_checked, r.pairs, r.cpu_pairs, r.n_overflow, r.max_stopping_time, r.errors)
    wide = (r.max_excursion, r.max_excursion_seed, r.max_stopping_time_seed, *r.overflow)
    return {"counts": np.array(head, dtype=np.int64),
            "numbers": np.frombuffer(b"".join(x.to_bytes(16, "little") for x in wide), dtype=np.int32)}


def run(s):
    kind = s["kind"]
    if kind == "range":
        return _ranges([s["v"].verify_range(*s["args"], negative=s["negative"])])
    if kind == "plan":
        s["plan"].launch()
        return _ranges(s["plan"].results())
    if kind == "batch":
        return _ranges(s["v"].verify_batch(s["reqs"]))
    if kind == "query":
        status, st, exc = s["v"].trajectory_array(s["seeds"])
        return {"status": status.view(np.int32), "stopping_time": st.view(np.int64), "excursion": exc.view(np.int32)}
    if kind == "line":
        return _case(s["v"].run_case(*s["line"], overflow_cap=1024))
    if kind == "lines":
        return _case(s["v"].run_cases(s["lines"], overflow_cap=1024, per_case=False)[0])
    if kind == "pairs":
        return _case(s["v"].launchkernel(s["bigindex"], s["pairs"], overflow_cap=1024))
    srv = s["server"]
    tickets = [srv.submit_range(*q) if isinstance(q, tuple) else srv.submit_trajectory_array(q) for q in s["reqs"]]
    answers = [srv.wait(t) for t in tickets]
    queries = [a for a in answers if a.range is None]
    out = {}
    if len(queries) < len(answers):
        out["ranges"] = _ranges([a.range for a in answers if a.range is not None])
    if queries:
        out["status"] = np.concatenate([a.traj_status for a in queries]).view(np.int32)
        out["stopping_time"] = np.concatenate([a.traj_stopping_time for a in queries]).view(np.int64)
        out["excursion"] = np.concatenate([a.traj_excursion for a in queries]).view(np.int32)
    return out


# ----------------------------------------------------------------------------
# work and values
# ----------------------------------------------------------------------------

# residues mod 2^k that survive the k-step descent sieve
SURVIVORS = {16: 2114, 20: 27328, 24: 286581, 34: 151917636}


def _range_work(size, k, bits, mod9=True):
    """Every surviving residue's entry read once (16 bytes, at most one per seed), request in, result
    out; per seed the k-step jump and four steps that find its descent, one multiply-add and one
    compare per limb each."""
    seeds = size * SURVIVORS[k] / 2.0 ** k * (5 / 9 if mod9 else 1.0)
    limbs = -(-(bits + 8) // 32)
    return {"bytes": 16.0 * min(seeds, SURVIVORS[k]) + 24 + 104, "flops": seeds * 10.0 * limbs}


def _mean_size(lo_log2, hi_log2):
    return (2.0 ** hi_log2 - 2.0 ** lo_log2) / ((hi_log2 - lo_log2) * math.log(2))


def _query_work(n):
    # seed in, results out; about 1000 steps of a 160-bit value in run pairs of four steps, two operations a limb
    return {"bytes": n * (32.0 + 76.0), "flops": n * 250 * 5 * 2 * 2.0}


def work(case):
    kind = case["kind"]
    if kind == "range":
        return _range_work(case["size"], case["k"], case["hi"], case.get("mod9", True))
    if kind in ("plan", "batch"):
        w = _range_work(case["n"] * _mean_size(case["lo_log2"], case["hi_log2"]), 24, 64)
        return {"bytes": w["bytes"] + case["n"] * 128.0, "flops": w["flops"]}
    if kind == "query":
        return _query_work(case["n"])
    if kind == "served":
        w = _range_work(0.7 * case["n"] * _mean_size(case["lo_log2"], case["hi_log2"]), 24, 64)
        q = _query_work(0.3 * case["n"] * _mean_size(0, 16))
        return {"bytes": w["bytes"] + q["bytes"] + 128.0 * case["n"], "flops": w["flops"] + q["flops"]}
    # cases mode: the whole tree at N has 2.326e10 seeds at N = 45, 7.67e7 at N = 36 and about 1.89 times
    # as many for each more bit; a seed takes 5 checkpoints of two run pairs, two operations a limb and run
    tree = 2.326e10 * 1.887 ** (case["maxbits"] - 45)
    if kind == "pairs":
        seeds, pairs = case["n"] * 100.0, float(case["n"])
    else:
        share = min(1.0, (case.get("n", 1)) / max(1, len(_split(case["maxbits"], case["cut"]))))
        seeds, pairs = tree * share, tree * share / 100.0
    return {"bytes": 32.0 * pairs + 33 * 64 * 1024, "flops": seeds * 5 * 2 * 2 * 2 * 2.0}


def _trajectory(n, negative=False):
    """(stopping time, excursion) of one seed in plain integers."""
    x, e, s = n, n, 0
    while True:
        x = (3 * x + (-1 if negative else 1)) >> 1 if x & 1 else x >> 1
        s += 1
        e = max(e, x)
        if x < n:
            return s, e


def _exact_range(off, size, k, mod9, negative):
    keep = ({0, 2, 3, 6, 8} if negative else {0, 1, 3, 6, 7}) if mod9 else set(range(9))
    r, seeds = cb.RangeResult(0, 0, 0, 0, 0, 0, 0), 0
    for n in range(max(off, 2), off + size):
        if n % 9 not in keep and not (negative and n == 5):
            continue
        if n >> k:  # the k-step descent sieve
            x, f, alive = n & ((1 << k) - 1), 0, True
            for j in range(1, k + 1):
                if x & 1:
                    x, f = (3 * x + (-1 if negative else 1)) >> 1, f + 1
                else:
                    x >>= 1
                if 3 ** f < 1 << j:
                    alive = False
                    break
            if not alive:
                continue
        seeds += 1
        s, e = _trajectory(n, negative)
        if s > r.max_stopping_time:
            r.max_stopping_time, r.max_stopping_time_seed = s, n
        if e > r.max_excursion:
            r.max_excursion, r.max_excursion_seed = e, n
    r.seeds_checked = seeds
    return _ranges([r])


def exact(case, seed):
    rng = random.Random(seed)
    if case["kind"] == "range" and case["size"] <= 1 << 21 and not (case.get("negative") and case["lo"] < 8):
        off = _offset(rng, case["lo"], case["hi"], case["align"])
        return _exact_range(off, case["size"], case["k"], case.get("mod9", True), case.get("negative", False))
    if case["kind"] == "query" and case["n"] <= 2048:
        x = _query_seeds(rng, case["n"])
        got = [_trajectory(sum(int(w) << (32 * j) for j, w in enumerate(row))) for row in x]
        exc = b"".join(e.to_bytes(64, "little") for _, e in got)
        return {"status": np.zeros(case["n"], dtype=np.int32), "stopping_time": np.array([s for s, _ in got], dtype=np.int64),
                "excursion": np.frombuffer(exc, dtype=np.int32).reshape(case["n"], 16)}
    return None
