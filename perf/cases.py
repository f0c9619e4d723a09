"""The work that programs have this library do, as measurable cases.

Every case goes through the public entry points of ``meikey_b200`` (``Context``, ``Job``,
``Graph``, ``Server``) the way a program calls them:

  derive   public keys of a range of indices, copied to the host (self-checks, audits,
           re-deriving found keys; the all-keys comparison of 2^20 seeds)
  search   launches of one job over a range and the candidates found there
  multi    64 text patterns and 8 regexes in one job, a CUDA-graph replay of its launches,
           and the lowest confirmed key of every needle
  serve    jobs arriving at a continuous-batching server until each one is answered
  find     one whole request: make a job, search until a key is found, release the job

A program keeps one ``Context`` (the comb table and the launch geometry) for its lifetime, and
a job while it searches with it; both are part of a case's state.  Keys, start indices and
needles come from the seed.
"""
import hashlib
import random

import numpy as np

import meikey_b200 as mk

ALPHABET = "ABCDEFGHIJKLMNOPQRSTUVWXYZabcdefghijklmnopqrstuvwxyz0123456789+/"

SOURCES = {"chacha20": mk.SEED_CHACHA20, "counter": mk.SEED_COUNTER, "incremental": mk.SEED_INCREMENTAL}

# regexes of the multi-pattern workload, DFAs of 6..57 states
REGEXES = ["(ab|cd|ef)[+/]x", "(?:aa|bb)(?:cc|dd)$", "x.{2}y.{2}z", "(?:ab|ba).{2}[0-9]{2}$",
           "z[0-9]{3}z", "(?:xyz|XYZ)$", "(?:AA|BB|CC)[0-9]{3}", "[ab].{4}[cd]z[0-9]"]

# budget of one served job and indices of one server tick, as the serving benchmark sets them
SERVE_BUDGET, SERVE_ITERS = 1 << 26, 8

# candidates a searching program makes room for; needles are short enough for a range to hold
# some and long enough for it to hold fewer than this
MAX_HITS = 8192


def context_options(rows=12, kpt=16, batch=0, rotates=False, ring=0):
    """A context's options as plain values of a case (the defaults are those of ``Context``)."""
    return {"rows": rows, "kpt": kpt, "batch": batch, "rotates": rotates, "ring": ring}


def listed():
    return [
        # a handful of keys: what a self-check or a tool that re-derives its keys asks for
        {"name": "derive_257", "kind": "derive", "source": "chacha20", "n": 257, "noalloc": False,
         **context_options()},
        # the same in the entry point that allocates nothing, an odd few thousand counter keys
        {"name": "derive_noalloc_4099", "kind": "derive", "source": "counter", "n": 4099, "noalloc": True,
         **context_options(kpt=8)},
        # an audit of an incremental run: consecutive points
        {"name": "derive_incremental_100003", "kind": "derive", "source": "incremental", "n": 100003,
         "noalloc": False, **context_options()},
        # the small secure workload: all keys of 2^20 seeds on the host
        {"name": "derive_2p20", "kind": "derive", "source": "chacha20", "n": 1 << 20, "noalloc": False,
         **context_options(kpt=8)},
        # the small secure workload's search: a 4-character case-insensitive needle, one iteration
        {"name": "search_small", "kind": "search", "source": "chacha20", "count": 1 << 20, "length": 4,
         "mode": "contains_ci", **context_options()},
        # the secure throughput workload: a case-sensitive needle, inversion batched over 256 keys
        {"name": "search_secure", "kind": "search", "source": "chacha20", "count": 1 << 29, "length": 5,
         "mode": "contains", **context_options(kpt=8, batch=256)},
        # the low-security counter mode with a case-insensitive needle
        {"name": "search_counter", "kind": "search", "source": "counter", "count": 1 << 27, "length": 5,
         "mode": "contains_ci", **context_options(kpt=8)},
        # the incremental workload: a case-sensitive suffix
        {"name": "search_incremental", "kind": "search", "source": "incremental", "count": 1 << 30, "length": 4,
         "mode": "suffix", **context_options()},
        # a short incremental search, an odd number of candidates and a frequent needle
        {"name": "search_incremental_short", "kind": "search", "source": "incremental", "count": 5_000_011,
         "length": 4, "mode": "contains", **context_options(kpt=8)},
        # the multi-pattern workload: 64 text needles and 8 regexes, four launches a graph replay
        {"name": "multi_72", "kind": "multi", "source": "chacha20", "count": 1 << 27, "text": 64, "regex": 8,
         "launches": 4, **context_options(kpt=16, batch=256, rotates=True, ring=1 << 22)},
        # a serving process: 40 jobs in two bursts, 4 to 8 characters, mixed modes
        {"name": "serve_40", "kind": "serve", "source": "chacha20", "jobs": 40, **context_options(kpt=8, ring=1 << 22)},
        # one request answered as fast as possible: a 4-character case-insensitive needle
        {"name": "find_4", "kind": "find", "source": "chacha20", "length": 4, "mode": "contains_ci", "iters": 1,
         **context_options()},
    ]


def log_uniform(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    kind = rng.choice(("derive", "derive", "search", "search", "search", "multi", "serve", "find"))
    source = rng.choice(("chacha20", "counter", "incremental"))
    rows, kpt = rng.choice((12, 12, 16)), rng.choice((4, 8, 16))
    if kind == "derive":
        noalloc = source != "incremental" and rng.random() < 0.4
        n = log_uniform(rng, 1, 60000) if noalloc else log_uniform(rng, 1, 1 << 20)
        return {"kind": kind, "source": source, "n": n, "noalloc": noalloc, **context_options(rows, kpt)}
    if kind == "search":
        count = log_uniform(rng, 1 << 20, (1 << 29) if source == "incremental" else (1 << 27))
        mode = rng.choice(("contains", "suffix", "contains_ci"))
        length = 1  # the longest needle that about eight candidates or more match
        while count * (1 if mode == "suffix" else 40) >= 8 * 64 ** (length + 1):
            length += 1
        return {"kind": kind, "source": source, "count": count, "length": length, "mode": mode,
                **context_options(rows, kpt, rotates=rng.random() < 0.2)}
    if kind == "multi":
        return {"kind": kind, "source": source, "count": log_uniform(rng, 1 << 23, 1 << 26),
                "text": rng.randint(2, 64), "regex": rng.randint(0, 8), "launches": rng.randint(1, 4),
                **context_options(rows, rng.choice((8, 16)), rotates=rng.random() < 0.7, ring=1 << 22)}
    if kind == "serve":
        return {"kind": kind, "source": "chacha20", "jobs": rng.randint(4, 48),
                **context_options(rows, kpt, ring=1 << 22)}
    return {"kind": kind, "source": source, "length": rng.choice((3, 4)),
            "mode": rng.choice(("contains", "contains_ci")), "iters": rng.randint(1, 4), **context_options(rows, kpt)}


def make_context(case):
    return mk.Context(device=0, table_rows=case["rows"], keys_per_thread=case["kpt"],
                      inversion_batch=case["batch"], inverter_rotates=case["rotates"], hit_capacity=case["ring"])


def inputs(case, seed):
    """(rng, key, first): the seed's random stream, the job key and the first index."""
    rng = random.Random(int(seed))
    key = bytearray(rng.randbytes(32))
    if case["source"] == "incremental":  # a clamped scalar, as a program takes from one seed
        key[0] &= 248
        key[31] = key[31] & 127 | 64
    return rng, bytes(key), rng.randrange(1 << 40)


def text_needle(rng, length, mode):
    text = "".join(rng.choice(ALPHABET) for _ in range(length))
    if mode == "suffix":
        return mk.Needle.suffix(text)
    return mk.Needle.contains(text, case_sensitive=mode == "contains")


def mixed_needles(rng, n, lo, hi):
    return [text_needle(rng, rng.randint(lo, hi), rng.choice(("contains", "suffix", "contains_ci"))) for _ in range(n)]


def prepare(case, seed):
    rng, key, first = inputs(case, seed)
    ctx = make_context(case)
    s = {"case": case, "ctx": ctx, "key": key, "source": SOURCES[case["source"]], "first": first}
    if case["kind"] == "search":
        s["iters"] = -(-case["count"] // ctx.keys_per_iter)
        s["job"] = ctx.job(key, s["source"], [text_needle(rng, case["length"], case["mode"])])
    elif case["kind"] == "multi":
        needles = mixed_needles(rng, case["text"], 3, 9)
        needles += [mk.Needle.regex(r, max_states=64) for r in REGEXES[:case["regex"]]]
        s["job"] = ctx.job(key, s["source"], needles)
        iters = max(1, -(-case["count"] // (ctx.keys_per_iter * case["launches"])))
        s["graph"] = s["job"].graph(iters, case["launches"])
    elif case["kind"] == "serve":
        s["needles"] = mixed_needles(rng, case["jobs"], 4, 8)
    elif case["kind"] == "find":
        s["needle"] = text_needle(rng, case["length"], case["mode"])
    return s


def key_array(keys):
    return np.frombuffer(b"".join(keys), dtype=np.uint8).reshape(-1, 32)


def run_derive(s):
    call = s["ctx"].derive_noalloc if s["case"]["noalloc"] else s["ctx"].derive
    return np.frombuffer(call(s["key"], s["source"], s["first"], s["case"]["n"]), dtype=np.uint8).reshape(-1, 32)


def run_search(s):
    """Candidates (index, needle) of the `count` indices from the first one, -1 behind the last."""
    s["job"].launch(s["first"], s["iters"])
    hits, _ = s["job"].hits(cap=MAX_HITS)
    end = s["first"] + s["case"]["count"]
    out = np.full((MAX_HITS, 2), -1, dtype=np.int64)
    for k, hit in enumerate(h for h in hits if h[0] < end):
        out[k] = hit
    return out


def run_multi(s):
    s["graph"].launch(s["first"])
    found = s["job"].first_matches()
    return {"index": np.array([m["index"] if m else -1 for m in found], dtype=np.int64),
            "pk": key_array(m["pk"] if m else bytes(32) for m in found),
            "secret": key_array(m["secret"] if m else bytes(32) for m in found)}


def run_serve(s):
    needles, results = s["needles"], {}
    half = len(needles) // 2
    with mk.Server(s["ctx"], s["key"], s["source"], max_jobs=128, iters_per_tick=SERVE_ITERS, budget=SERVE_BUDGET,
                   hit_capacity=1 << 21, first=s["first"]) as srv:
        for i, n in enumerate(needles[:half]):
            srv.submit(n, i)
        srv.tick()
        for i, n in enumerate(needles[half:]):
            srv.submit(n, half + i)
        while len(results) < len(needles):
            srv.tick()
            results.update((r["id"], r) for r in srv.results())
    ordered = [results[i] for i in range(len(needles))]
    return {"index": np.array([r["index"] if r["found"] else -1 for r in ordered], dtype=np.int64),
            "pk": key_array(r["pk"] for r in ordered), "secret": key_array(r["secret"] for r in ordered)}


def run_find(s):
    with s["ctx"].job(s["key"], s["source"], [s["needle"]]) as job:
        r = job.search(first=s["first"], max_tries=1 << 28, iters=s["case"]["iters"])
    return {"index": r["index"] if r["found"] else -1, "pk": key_array([r["pk"]]), "secret": key_array([r["secret"]])}


def run(state):
    return {"derive": run_derive, "search": run_search, "multi": run_multi, "serve": run_serve,
            "find": run_find}[state["case"]["kind"]](state)


# Integer operations a key costs: limb products of the field multiplications (64 multiply-adds
# each) and the hash.  A hashed key takes a mixed addition (7 multiplications) per comb row but
# the first and the last (3), and the batched inversion (4); a consecutive point takes about
# half a mixed addition and the inversion.
MUL_OPS, HASH_OPS = 128, 4800


def keys_of(case):
    if case["kind"] == "derive":
        return case["n"]
    if case["kind"] in ("search", "multi"):
        return case["count"]
    if case["kind"] == "serve":  # most batches hold a job that takes the whole budget
        return SERVE_BUDGET
    # find: positions of the needle against its 64-value characters (about two values each when
    # the case does not matter), with both values of one sign-dependent character
    values = 64 / (52 / 32 if case["mode"] == "contains_ci" else 1)
    return max(1, int(values ** case["length"] / (44 - case["length"])))


def work(case):
    keys = keys_of(case)
    rows = case["rows"]
    if case["source"] == "incremental":
        ops, bytes_ = 6 * MUL_OPS, 0
    else:
        ops, bytes_ = (7 * (rows - 2) + 3 + 4) * MUL_OPS + HASH_OPS, 96 * rows
    if case["kind"] == "derive":
        ops, bytes_ = ops + 4 * MUL_OPS, bytes_ + 32
    return {"bytes": float(bytes_ * keys + 1), "flops": float(ops * keys)}


# ---------------------------------------------------------------------------
# the derived keys again, in plain Python integers
# ---------------------------------------------------------------------------

P = 2**255 - 19
D = -121665 * pow(121666, -1, P) % P


def base_point():
    y = 4 * pow(5, -1, P) % P
    u, v = (y * y - 1) % P, (D * y * y + 1) % P
    x = u * v**3 * pow(u * v**7, (P - 5) // 8, P) % P
    if (v * x * x - u) % P:
        x = x * pow(2, (P - 1) // 4, P) % P
    return (P - x if x & 1 else x), y


def point_add(a, b):
    """a + b in extended coordinates (X, Y, Z, T), twisted Edwards with a = -1 (complete)."""
    A, B = (a[1] - a[0]) * (b[1] - b[0]), (a[1] + a[0]) * (b[1] + b[0])
    C, Z = 2 * D * a[3] * b[3] % P, 2 * a[2] * b[2]
    E, F, G, H = (B - A) % P, (Z - C) % P, (Z + C) % P, (B + A) % P
    return E * F % P, G * H % P, F * G % P, E * H % P


def window_table():
    """table[w][d] = d · 256^w · B."""
    x, y = base_point()
    step, table = (x, y, 1, x * y % P), []
    for _ in range(32):
        row = [(0, 1, 1, 0)]
        for _ in range(256):
            row.append(point_add(row[-1], step))
        table.append(row[:256])
        step = row[256]
    return table


def compress(points):
    prefix, run_ = [], 1
    for p in points:
        prefix.append(run_)
        run_ = run_ * p[2] % P
    inv, out = pow(run_, -1, P), []
    for p, pre in zip(reversed(points), reversed(prefix)):
        zi = inv * pre % P
        inv = inv * p[2] % P
        out.append(((p[1] * zi % P) | ((p[0] * zi % P & 1) << 255)).to_bytes(32, "little"))
    return out[::-1]


def chacha20_block(key, counter):
    """Block `counter` of the ChaCha20 keystream (RFC 8439 rounds, 64-bit counter, nonce 0)."""
    mask = 0xFFFFFFFF
    init = [0x61707865, 0x3320646E, 0x79622D32, 0x6B206574]
    init += [int.from_bytes(key[4 * i:4 * i + 4], "little") for i in range(8)]
    init += [counter & mask, counter >> 32, 0, 0]
    s = list(init)
    for _ in range(10):
        for a, b, c, d in ((0, 4, 8, 12), (1, 5, 9, 13), (2, 6, 10, 14), (3, 7, 11, 15),
                           (0, 5, 10, 15), (1, 6, 11, 12), (2, 7, 8, 13), (3, 4, 9, 14)):
            for x, y, z, n in ((a, b, d, 16), (c, d, b, 12), (a, b, d, 8), (c, d, b, 7)):
                s[x] = (s[x] + s[y]) & mask
                t = s[z] ^ s[x]
                s[z] = (t << n | t >> (32 - n)) & mask
    return b"".join(((s[i] + init[i]) & mask).to_bytes(4, "little") for i in range(16))


def scalar(case, key, index):
    if case["source"] == "incremental":
        return int.from_bytes(key, "little") + index
    if case["source"] == "counter":
        tail = (int.from_bytes(key[24:], "little") + index) % 2**64
        seed = key[:24] + tail.to_bytes(8, "little")
    else:
        seed = chacha20_block(key, index >> 1)[32 * (index & 1):][:32]
    h = int.from_bytes(hashlib.sha512(seed).digest()[:32], "little")
    return h & (2**254 - 8) | 2**254


def exact(case, seed):
    if case["kind"] != "derive" or case["n"] > 20000:
        return None  # other results are indices of matching keys, or too many keys to recompute here
    _, key, first = inputs(case, seed)
    table, points = window_table(), []
    for index in range(first, first + case["n"]):
        p = (0, 1, 1, 0)
        for w, d in enumerate(scalar(case, key, index).to_bytes(32, "little")):
            if d:
                p = point_add(p, table[w][d])
        points.append(p)
    return key_array(compress(points))
