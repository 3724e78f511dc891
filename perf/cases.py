"""The work that programs have this framework do, as cases that can be timed.

Paths (a case's "path"):
  single      one generator fills a buffer the caller keeps, once per entry of
              "kinds" (the reference's mtgp*_init + genrand_* loops)
  bank        one generator per parameter set, the same number of values each,
              by Pool.fill (the shape of the reference's CUDA samples)
  bank_plan   the same values through a plan that the program made once
  batch       uneven requests of many jumped substreams through a plan
  submit      a list of short requests of mixed kinds handed over per call
  substreams  a program's start: a pool of jumped substreams and its first
              draws
  polys       jump polynomials of arbitrary distances
  skip        one generator jumps ahead by an arbitrary distance and draws
  serve       a burst of requests through the continuous-batching server

Sizes are those of the tests and of bench.py (2^20 pairs, banks of 128 and 200
sets, 4096 substreams, lognormal request lengths, 4096 polynomials) or generic
ones around them, odd ones among them.
"""
import os

import numpy as np
import torch

from mtgp_gb300.api import (MTGP32, MTGP64, Pool, REQUEST_DTYPE, Server, work_items)
from mtgp_gb300.params import DATA, TABLES, jump_table, load_table

# kind numbers: 0 integer, 1 [1,2), 2 [0,1), 3 (0,1], 4 (0,1)
JUMPED = {32: "mtgp32_fast_11213", 64: "mtgp64dc_fast_11213"}  # sets with a shipped jump table


def listed():
    return [
        # a program that draws a handful of numbers at a time: latency
        {"name": "single_u32_1000", "path": "single", "table": "mtgp32_fast_11213", "set": 0,
         "n": 1000, "kinds": "0", "offset": 0},
        # one ordinary array of floats from one generator, into a slice that
        # is not vector-aligned
        {"name": "single_f32_200003", "path": "single", "table": "mtgp32_fast_11213", "set": 5,
         "n": 200003, "kinds": "2", "offset": 1},
        # the smallest documented benchmark: 2^20 integers, then 2^20 floats
        {"name": "single_pair_2p20", "path": "single", "table": "mtgp32_fast_11213", "set": 0,
         "n": 1 << 20, "kinds": "01", "offset": 0},
        # one large array of doubles from one generator, a ragged size
        {"name": "single_f64_33542087", "path": "single", "table": "mtgp64dc_fast_11213", "set": 3,
         "n": 33542087, "kinds": "1", "offset": 0},
        # the reference sample's shape: 128 sets, one fill for all
        {"name": "bank_u32_128x2p21", "path": "bank", "table": "mtgp32_fast_11213", "sets": 128,
         "n": 1 << 21, "kind": 0},
        # the 64-bit bank of 200 sets through a kept plan
        {"name": "bank_plan_u64_200x2p20", "path": "bank_plan", "table": "mtgp64dc_fast_11213",
         "sets": 200, "n": 1 << 20, "kind": 0},
        # the headline workload: 4096 substreams, lognormal request lengths
        {"name": "batch_u32_4096_lognormal", "path": "batch", "bits": 32, "streams": 4096,
         "median": 65536, "kind": 0},
        # many short requests of integers and floats, planned on each call
        {"name": "submit_mixed_2000", "path": "submit", "bits": 32, "streams": 1000,
         "requests": 2000, "median": 1500},
        # what a simulation does once at its start
        {"name": "substreams_4096", "path": "substreams", "bits": 32, "streams": 4096, "n": 256},
        # distances of a work distribution turned into polynomials
        {"name": "polys_1000", "path": "polys", "bits": 32, "count": 1000},
        # a worker moves to its place in one long stream
        {"name": "skip_2p50", "path": "skip", "bits": 32, "log2_steps": 50, "n": 1000},
        # a burst of clients' requests on the server
        {"name": "serve_burst_4000", "path": "serve", "requests": 4000, "median": 16384},
    ]


def _log(rng, lo, hi):
    """A whole number between lo and hi, spread over its logarithm."""
    return max(lo, min(hi, int(round(lo * (hi / lo) ** rng.random()))))


def draw(rng):
    path = rng.choice(["single", "single", "single", "bank", "bank_plan", "batch", "submit",
                       "substreams", "polys", "skip", "serve"])
    bits = rng.choice([32, 32, 64])
    if path == "single":
        table = rng.choice(sorted(t for t in TABLES if t.startswith("mtgp%d" % bits)))
        long_ok = table.endswith(("11213", "23209"))
        return {"path": path, "table": table, "set": rng.randrange(TABLES[table][1]),
                "n": _log(rng, 1, 1 << (25 if long_ok else 19)),
                "kinds": rng.choice("01234"), "offset": rng.randrange(4)}
    if path in ("bank", "bank_plan"):
        table = rng.choice(sorted(t for t in TABLES if t.startswith("mtgp%d" % bits)))
        if path == "bank_plan" and not table.endswith("11213"):
            table = JUMPED[bits]  # the long exponents' tables take too long to be made here
        sets = _log(rng, 2, TABLES[table][1] if path == "bank" else 64)
        return {"path": path, "table": table, "sets": sets,
                "n": _log(rng, 1000, (1 << 21) // (bits // 32)), "kind": rng.randrange(5)}
    if path == "batch":
        return {"path": path, "bits": bits, "streams": _log(rng, 16, 4096 if bits == 32 else 1024),
                "median": _log(rng, 500, 60000), "kind": rng.randrange(5)}
    if path == "submit":
        return {"path": path, "bits": bits, "streams": _log(rng, 4, 1000),
                "requests": _log(rng, 4, 4000), "median": _log(rng, 50, 5000)}
    if path == "substreams":
        return {"path": path, "bits": bits, "streams": _log(rng, 2, 4096), "n": _log(rng, 1, 1000)}
    if path == "polys":
        return {"path": path, "bits": bits, "count": _log(rng, 1, 4096)}
    if path == "skip":
        return {"path": path, "bits": bits, "log2_steps": rng.randrange(23, 63),
                "n": _log(rng, 1, 20000)}
    return {"path": path, "requests": _log(rng, 16, 4000), "median": _log(rng, 1000, 16384)}


def _bits(c):
    return c["bits"] if "bits" in c else 32 if c.get("table", "mtgp32").startswith("mtgp32") else 64


def _buffer(bits, kind, n):
    dt = {(32, 0): torch.int32, (32, 1): torch.float32,
          (64, 0): torch.int64, (64, 1): torch.float64}[bits, min(int(kind), 1)]
    return torch.empty(int(n), dtype=dt, device="cuda")


def _rng(seed):
    return np.random.default_rng([int(seed), 20])


def _lognormal(rng, median, n):
    return np.clip(np.rint(rng.lognormal(np.log(median), 1.0, n)), 1, 2 ** 22).astype(np.int64)


def _sizes(case, n):
    """The requests' lengths and a uniform number each: the same for every
    seed, so that a case's outputs have one shape."""
    rng = np.random.default_rng(42)
    return _lognormal(rng, case["median"], n), rng.random(n)


def _distances(rng, log2, n):
    return [int(x) for x in rng.integers(1 << (log2 - 1), 1 << log2, n, dtype=np.uint64)]


def prepare(case, seed):
    c, path, rng, bits = case, case["path"], _rng(seed), _bits(case)
    gseed = int(rng.integers(1, 2 ** 31))
    st = {"path": path}
    if path == "single":
        gen = (MTGP32 if bits == 32 else MTGP64)(load_table(c["table"])[c["set"]], seed=gseed)
        st["gen"] = gen
        st["fills"] = []
        for k in c["kinds"]:
            buf = _buffer(bits, k, c["n"] + c["offset"])
            st["fills"].append((int(k), buf[c["offset"]:]))
    elif path in ("bank", "bank_plan"):
        tab = load_table(c["table"])
        m, n = c["sets"], c["n"]
        pool = Pool.create([tab[i] for i in range(m)], rng.integers(1, 2 ** 31, m))
        st.update(pool=pool, out=_buffer(bits, c["kind"], m * n), kind=c["kind"], n=n)
        if path == "bank_plan":
            st["plan"] = pool.plan(work_items(range(m), [c["kind"]] * m, [n] * m,
                                              [i * n * (bits // 8) for i in range(m)]))
    elif path == "batch":
        m = c["streams"]
        pool = Pool.substreams(load_table(JUMPED[bits])[0], gseed, m, jump_table(bits))
        lens, _ = _sizes(c, m)
        offs = (np.cumsum(lens) - lens) * (bits // 8)
        st.update(pool=pool, out=_buffer(bits, c["kind"], lens.sum()),
                  plan=pool.plan(work_items(range(m), [c["kind"]] * m, lens, offs)))
    elif path == "submit":
        m, r = c["streams"], c["requests"]
        tab = load_table(JUMPED[bits])
        pool = Pool.create(list(tab[0:16]), rng.integers(1, 2 ** 31, m), np.arange(m) % 16)
        lens, _ = _sizes(c, r)
        offs = (np.cumsum(lens) - lens) * (bits // 8)
        # a tenth of the requests leave out a few of their stream's values
        skips = np.where(rng.random(r) < 0.1, rng.integers(1, 500, r), 0)
        st.update(pool=pool, out=_buffer(bits, 0, lens.sum()),
                  items=work_items(rng.integers(0, m, r), rng.choice([0, 1, 2], r), lens, offs,
                                   skips))
    elif path == "substreams":
        st.update(params=load_table(JUMPED[bits])[0], seed=gseed, table=jump_table(bits),
                  count=c["streams"], n=c["n"], out=_buffer(bits, 0, c["streams"] * c["n"]))
    elif path == "polys":
        pool = Pool.create([load_table(JUMPED[bits])[0]], [gseed])
        st.update(pool=pool, steps=rng.integers(1 << 40, 1 << 63, c["count"], dtype=np.uint64))
    elif path == "skip":
        gen = (MTGP32 if bits == 32 else MTGP64)(load_table(JUMPED[bits])[0], seed=gseed)
        st.update(gen=gen, steps=_distances(rng, c["log2_steps"], 256), at=0,
                  out=_buffer(bits, 0, c["n"]))
    elif path == "serve":
        # 512 32-bit and 64 64-bit substreams; integers, floats and 64-bit
        # integers 60/30/10, a tenth of the requests at an offset 2^17..2^40
        r = c["requests"]
        a = Pool.substreams(load_table(JUMPED[32])[0], gseed, 512, jump_table(32))
        b = Pool.substreams(load_table(JUMPED[64])[0], gseed, 64, jump_table(64))
        req = np.zeros(r, dtype=REQUEST_DTYPE)
        req["count"], u = _sizes(c, r)
        req["pool"] = u >= 0.9
        req["kind"] = np.where((u >= 0.6) & (u < 0.9), 2, 0)
        req["stream"] = np.where(u < 0.9, rng.integers(0, 512, r), rng.integers(0, 64, r))
        req["skip"] = np.where(rng.random(r) < 0.1,
                               np.left_shift(1, rng.integers(17, 41, r)), 0)
        outs = []
        for p, w in ((0, 32), (1, 64)):
            mine = req["pool"] == p
            lens = req["count"][mine].astype(np.int64)
            out = _buffer(w, 0, lens.sum() + 1)
            req["dst"][mine] = out.data_ptr() + (np.cumsum(lens) - lens) * (w // 8)
            outs.append(out[:int(lens.sum())])
        st.update(server=Server(a, b, budget_bytes=2 << 30, slots=4, max_batch=4096),
                  requests=req, arrivals=np.zeros(r), outs=outs)
    else:
        raise ValueError(path)
    return st


def run(state):
    st, path = state, state["path"]
    if path == "single":
        return [st["gen"].fill_into(kind, out) for kind, out in st["fills"]]
    if path == "bank":
        st["pool"].fill(st["kind"], st["out"], st["n"])
        return st["out"]
    if path in ("bank_plan", "batch"):
        st["plan"].launch(st["out"])
        return st["out"]
    if path == "submit":
        st["pool"].submit(st["items"], st["out"])
        return st["out"]
    if path == "substreams":
        pool = Pool.substreams(st["params"], st["seed"], st["count"], st["table"])
        pool.fill(0, st["out"], st["n"])
        pool.close()
        return st["out"]
    if path == "polys":
        return st["pool"].jump_polys(0, st["steps"])
    if path == "skip":
        st["gen"].jump_steps(st["steps"][st["at"] % len(st["steps"])])
        st["at"] += 1
        return st["gen"].fill_into(0, st["out"])
    st["server"].replay(st["requests"], st["arrivals"])
    return st["outs"]


def _lognormal_mean(median):
    return median * float(np.exp(0.5))


def work(case):
    """Bytes: outputs once, stream windows read and written once.  Flops:
    32-bit word operations, 12 a word generated (the recursion and the
    tempering; two lookups) and N * mexp / 2 XORs a jump; a product of
    polynomials counts as the XORs of half its shifted rows."""
    c, path, bits = case, case["path"], _bits(case)
    wb, half = bits // 8, bits // 32
    mexp = int(c["table"].split("_")[-1]) if "table" in c else 11213
    window = (mexp // bits + 1) * wb
    jump = (mexp // 32 + 1) * mexp / 2
    if path == "single":
        values, streams, extra = c["n"] * len(c["kinds"]), 1, 0
    elif path in ("bank", "bank_plan"):
        values, streams, extra = c["n"] * c["sets"], c["sets"], 0
    elif path == "batch":
        values, streams, extra = c["streams"] * _lognormal_mean(c["median"]), c["streams"], 0
    elif path == "submit":
        values, streams, extra = c["requests"] * _lognormal_mean(c["median"]), c["streams"], 0
    elif path == "substreams":
        values, streams, extra = c["streams"] * c["n"], c["streams"], c["streams"] * jump
    elif path == "polys":
        poly = (mexp // 32 + 1) * 4
        return {"bytes": c["count"] * (poly + 8), "flops": c["count"] * 7 * 2 * jump}
    elif path == "skip":
        values, streams, extra = c["n"], 1, jump
    else:
        mean = c["requests"] * _lognormal_mean(c["median"])
        return {"bytes": mean * (0.9 * 4 + 0.1 * 8), "flops": mean * 1.1 * 12}
    return {"bytes": values * wb + 2 * streams * window, "flops": values * 12 * half + extra}


# ---- what the values are, from the recursion alone -------------------------

def _params(table, k):
    """Parameter set k of a table file as plain numbers and arrays."""
    bits = 32 if table.startswith("mtgp32") else 64
    w = "<u%d" % (bits // 8)
    dt = np.dtype([("mexp", "<i4"), ("pos", "<i4"), ("sh1", "<i4"), ("sh2", "<i4"),
                   ("tbl", w, 16), ("tmp", w, 16), ("flt", w, 16), ("mask", w),
                   ("sha", "u1", 21), ("pad", "u1", 3)])
    return bits, np.fromfile(os.path.join(DATA, table + ".bin"), dtype=dt)[k]


def _seeded(bits, p, seed):
    n, m = int(p["mexp"]) // bits + 1, (1 << bits) - 1
    hidden = (int(p["tbl"][4]) ^ (int(p["tbl"][8]) << 16)) & m
    f = hidden if bits == 32 else hidden >> 32
    f = (f + (f >> 16)) & m
    f = (f + (f >> 8)) & 0xff
    fill = f * (0x01010101 if bits == 32 else 0x0101010101010101)
    mul, shr = (1812433253, 30) if bits == 32 else (6364136223846793005, 62)
    w = [seed]
    for k in range(1, n):
        w.append((hidden if k == 1 else fill) ^ ((mul * (w[-1] ^ (w[-1] >> shr)) + k) & m))
    return np.array(w, dtype="<u%d" % (bits // 8))


def _sequence(bits, p, window, n):
    """The window followed by the next n words of the recursion."""
    size, pos = len(window), int(p["pos"])
    seq = np.empty(size + n, dtype=window.dtype)
    seq[:size] = window
    tbl, mask = p["tbl"].astype(window.dtype), p["mask"].astype(window.dtype)
    sh1, sh2 = np.uint32(p["sh1"]), np.uint32(p["sh2"])
    for i in range(0, n, size - pos):
        m = min(size - pos, n - i)
        x = (seq[i:i + m] & mask) ^ seq[i + 1:i + 1 + m]
        y = seq[i + pos:i + pos + m]
        if bits == 32:
            r = x ^ (x << sh1) ^ (y >> sh2)
            seq[size + i:size + i + m] = r ^ tbl[r & 15]
        else:
            x, y = x.view("<u4"), y.view("<u4")  # low, high halves in turn
            x = x ^ (x << sh1)
            r = np.empty(2 * m, dtype="<u4")
            r[0::2] = x[1::2] ^ (y[0::2] >> sh2)
            r[1::2] = x[0::2] ^ (y[1::2] >> sh2)
            seq[size + i:size + i + m] = r.view("<u8") ^ tbl[r[0::2] & 15]
    return seq


def _temper(bits, p, seq, size, n, kind):
    r, t = seq[size:size + n], seq[int(p["pos"]) - 1:int(p["pos"]) - 1 + n].astype("<u4")
    t = t ^ (t >> np.uint32(16))
    t = (t ^ (t >> np.uint32(8))) & np.uint32(15)
    if kind == 0:
        return (r ^ p["tmp"][t]).view("<i%d" % (bits // 8))
    one = r.dtype.type(1)
    v = r >> r.dtype.type(9 if bits == 32 else 12)
    if kind == 4 and bits == 64:
        v = v | one
    v = v ^ p["flt"][t]
    if kind == 4 and bits == 32:
        v = v | one
    f = v.view("<f%d" % (bits // 8))
    return f if kind == 1 else f.dtype.type(2) - f if kind == 3 else f - f.dtype.type(1)


def _jumped(bits, p, window, steps):
    """The window `steps` values later: X^steps mod the characteristic
    polynomial (as a whole number, bit i = coefficient of X^i), applied."""
    with open(os.path.join(DATA, "mtgp%d_char_11213.txt" % bits)) as f:
        digits = f.read().strip()  # lowest coefficients first
    chi = int(digits[::-1], 16)
    deg = chi.bit_length() - 1
    r = 1
    for b in bin(steps)[2:]:
        r = int(bin(r)[2:], 4)  # the square: each bit to twice its place
        r <<= int(b)
        while r.bit_length() > deg:
            r ^= chi << (r.bit_length() - 1 - deg)
    seq = _sequence(bits, p, window, deg)
    out = np.zeros_like(window)
    for i in range(r.bit_length()):
        if (r >> i) & 1:
            out ^= seq[i:i + len(window)]
    return out


def exact(case, seed):
    """Computed from the recursion with numpy where one generator is at work;
    the other paths return words."""
    c, path, rng, bits = case, case["path"], _rng(seed), _bits(case)
    gseed = int(rng.integers(1, 2 ** 31))
    if path == "single":
        _, p = _params(c["table"], c["set"])
        window, got = _seeded(bits, p, gseed), []
        for k in c["kinds"]:
            seq = _sequence(bits, p, window, c["n"])
            got.append(_temper(bits, p, seq, len(window), c["n"], int(k)))
            window = seq[c["n"]:]
        return got
    if path == "skip":
        _, p = _params(JUMPED[bits], 0)
        window = _seeded(bits, p, gseed)
        window = _jumped(bits, p, window, _distances(rng, c["log2_steps"], 256)[0])
        seq = _sequence(bits, p, window, c["n"])
        return _temper(bits, p, seq, len(window), c["n"], 0)
    return None
