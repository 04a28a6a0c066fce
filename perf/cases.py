"""Performance cases of the library's public entry points.

Every case is one pass of work a caller gives the library: batched calls on a
map or a set, a queue of mixed batches, a key-value store with variable-size
values, a run of the serving loop.  Inputs are made on the GPU from a seed
(SplitMix64 counters and Gray et al.'s Zipf sampler, as in
lslab_b200.workload), so preparing a table of 2^27 keys takes well under a
second.  A pass leaves a table with the contents it found (puts overwrite the
same keys, temporary entries are removed again), so passes can be repeated and
each returns the same results.

Results are stored words, found bits and bytes, never computed numbers, so
there is no 64-bit reference value for any of them (exact() is None).
"""
from __future__ import annotations

import math

import torch

import lslab_b200 as L
from lslab_b200 import workload as W

_GOLDEN = 0x9E3779B97F4A7C15
_M1, _M2 = 0xBF58476D1CE4E5B9, 0x94D049BB133111EB
_CHUNK = 1 << 24  # prefill keys made and inserted at a time

# streams of one seed
_KEYS, _NEW, _TYPES, _RANKS, _VALUES, _SIZES, _BYTES, _HITS = range(1, 9)


# ------------------------------------------------------------------- cases
def listed():
    return [
        # a request handler looks up a few hundred keys at once in a small
        # table: one launch, latency is everything
        {"name": "get_500", "kind": "get", "log2": 16, "load": 16, "n": 500, "hit": 0.5,
         "theta": 0.0, "width": 64},
        # a small batch of short-lived entries (sessions, locks): put, later
        # removed; two calls, each with its grouping and ordering steps
        {"name": "temporary_777", "kind": "temporary", "log2": 16, "load": 16, "n": 777},
        # the reference's plain method at small size: 2^16 buckets, 2^20 keys,
        # 2^16 gets, half of them present; the table fits L2
        {"name": "get_65536", "kind": "get", "log2": 16, "load": 16, "n": 65536, "hit": 0.5,
         "theta": 0.0, "width": 64},
        # the read half of the 95/5 workload: 2^22 buckets, 2^26 keys, Zipf
        # 0.99; the table is far larger than L2
        {"name": "get_zipf_996147", "kind": "get", "log2": 22, "load": 16, "n": 996147,
         "hit": 1.0, "theta": 0.99, "width": 64},
        # the write half of the same batch, as a put call of its own
        {"name": "put_zipf_52429", "kind": "put", "log2": 22, "load": 16, "n": 52429,
         "theta": 0.99, "width": 64},
        # the whole 95/5 batch as one mixed call, gets before puts, in the
        # two-stream window form that the integration guide names for it
        {"name": "mixed_95_5", "kind": "mixed", "log2": 22, "load": 16, "n": 1 << 20,
         "get": 0.95, "put": 0.05, "update": 0.0, "sorted": True, "theta": 0.99, "form": "fused",
         "overlap": True},
        # a request queue's worth of mixed ops in arrival order (the size of
        # the serving loop's waves), an odd count
        {"name": "mixed_20011", "kind": "mixed", "log2": 20, "load": 8, "n": 20011,
         "get": 0.5, "put": 0.35, "update": 0.1, "sorted": False, "theta": 0.99, "form": "fused",
         "overlap": False},
        # 4096 small batches of uneven (lognormal) sizes placed back to back,
        # drained by one captured launch: 80/15/5 over 2^27 keys, 2^24 buckets
        {"name": "queue_4096", "kind": "queue", "log2": 24, "load": 8, "batches": 4096,
         "median": 512, "theta": 0.99},
        # a set that fits L2, one key per slot, 2^18-op batches 50/40/10
        # contains/insert/remove as one mixed call
        {"name": "set_mixed_262144", "kind": "set", "log2": 18, "load": 28, "n": 1 << 18,
         "form": "fused"},
        # a deduplication window over a large set by the per-op-type calls:
        # check keys, add the new ones, drop the expired ones
        {"name": "set_calls_130001", "kind": "set", "log2": 23, "load": 14, "n": 130001,
         "form": "calls"},
        # a key-value store whose clients overwrite and read values, then its
        # upkeep: the heap is compacted once the garbage is as large as the data
        {"name": "kv_32768", "kind": "kv", "log2": 12, "keys": 32768, "puts": 8192,
         "reads": 32768, "rounds": 4, "median": 128},
        # the serving loop with a full queue: requests of 1..4096 ops, 50/50
        # get/put, from the host's arena and back
        {"name": "serve_400", "kind": "serve", "log2": 20, "load": 8, "requests": 400,
         "max_ops": 4096},
    ]


def _log(rng, lo, hi):
    """An integer between lo and hi, spread over its logarithm."""
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["get", "get", "put", "temporary", "mixed", "mixed", "queue", "set", "set",
                       "kv", "serve"])
    log2 = rng.randint(10, 22)
    load = rng.choice([4, 8, 16, 24])
    theta = rng.choice([0.0, 0.99])
    if kind == "get":
        return {"kind": kind, "log2": log2, "load": load, "n": _log(rng, 1, 1 << 20),
                "hit": rng.choice([0.0, 0.5, 0.9, 1.0]), "theta": theta,
                "width": rng.choice([64, 64, 32])}
    if kind == "put":
        return {"kind": kind, "log2": log2, "load": load, "n": _log(rng, 1, 1 << 20),
                "theta": theta, "width": rng.choice([64, 64, 32])}
    if kind == "temporary":
        return {"kind": kind, "log2": log2, "load": min(load, 16),
                "n": min(_log(rng, 1, 1 << 18), 8 << log2)}
    if kind == "mixed":
        get, put, update = rng.choice([(0.95, 0.05, 0.0), (0.8, 0.15, 0.0), (0.5, 0.5, 0.0),
                                       (0.5, 0.3, 0.1), (0.2, 0.6, 0.1)])
        return {"kind": kind, "log2": log2, "load": load, "n": _log(rng, 64, 1 << 20),
                "get": get, "put": put, "update": update, "sorted": rng.random() < 0.5,
                "theta": theta, "form": rng.choice(["fused", "calls"]),
                "overlap": rng.random() < 0.25}
    if kind == "queue":
        return {"kind": kind, "log2": log2, "load": load, "batches": _log(rng, 16, 4096),
                "median": rng.choice([64, 256, 512]), "theta": theta}
    if kind == "set":
        return {"kind": kind, "log2": log2, "load": rng.choice([7, 14, 28, 56, 112]) if
                log2 < 20 else rng.choice([7, 14, 28]), "n": min(_log(rng, 64, 1 << 18), 7 << log2),
                "form": rng.choice(["fused", "calls"])}
    if kind == "kv":
        keys = _log(rng, 256, 32768)
        return {"kind": kind, "log2": max(4, keys.bit_length() - 4), "keys": keys,
                "puts": rng.randint(keys // 8, keys // 4), "reads": _log(rng, 64, 32768),
                "rounds": rng.randint(1, 4), "median": rng.choice([16, 64, 128])}
    return {"kind": "serve", "log2": rng.randint(12, 20), "load": rng.choice([4, 8, 16]),
            "requests": rng.randint(20, 400), "max_ops": rng.choice([64, 512, 4096])}


# ------------------------------------------------------------------ inputs
def _i64(x):
    """A 64-bit constant as torch's signed integer."""
    x &= (1 << 64) - 1
    return x - (1 << 64) if x >> 63 else x


def _shr(x, s):
    return (x >> s) & ((1 << (64 - s)) - 1)


def _mix(x):
    """SplitMix64's finaliser of a tensor of int64 counters times the golden ratio."""
    x = (x ^ _shr(x, 30)) * _i64(_M1)
    x = (x ^ _shr(x, 27)) * _i64(_M2)
    return x ^ _shr(x, 31)


def _stream(seed, what, count, start=0):
    i = torch.arange(start + 1, start + count + 1, dtype=torch.int64, device="cuda")
    return _mix(i * _i64(_GOLDEN) + _i64((seed + 1) * 0x51_7CC1_B727_2205 + what * 0x2545_F491_4F6C_DD1D))


def _at(seed, what, index):
    """Elements `index` of a stream."""
    return _mix((index + 1) * _i64(_GOLDEN) +
                _i64((seed + 1) * 0x51_7CC1_B727_2205 + what * 0x2545_F491_4F6C_DD1D))


def _uniform(seed, what, count):
    return _shr(_stream(seed, what, count), 11).double() * 2.0 ** -53


def _ranks(seed, items, theta, count, what=_RANKS):
    """Ranks in [0, items): uniform, or Zipf(theta) with rank 0 the most frequent."""
    u = _uniform(seed, what, count)
    if theta == 0.0:
        return (u * items).long().clamp_(0, items - 1)
    zn = W.zeta(items, theta)
    z2 = 1.0 + 0.5 ** theta
    eta = (1.0 - (2.0 / items) ** (1.0 - theta)) / (1.0 - z2 / zn)
    r = torch.floor(items * (eta * u - eta + 1.0) ** (1.0 / (1.0 - theta)))
    r = torch.where(u * zn < 1.0, torch.zeros_like(r),
                    torch.where(u * zn < z2, torch.ones_like(r), r))
    return r.long().clamp_(0, items - 1)


def _filled_map(case, seed):
    """A map of `load` keys per bucket (stream _KEYS, values key ^ constant)."""
    items = case["load"] << case["log2"]
    m = L.Map(case["log2"], ((1 << case["log2"]) * max(1, case["load"] // 8)) // 4 + 8192)
    for at in range(0, items, _CHUNK):
        k = _stream(seed, _KEYS, min(_CHUNK, items - at), at)
        v = k ^ _i64(W.VALUE_XOR)
        if case.get("width") == 32:
            v = v.int()
            L.lib().lsb_map_put_v32(m.handle, k.data_ptr(), v.data_ptr(), None, k.numel(),
                                    torch.cuda.current_stream().cuda_stream)
        else:
            m.put(k, v)
    return m, items


def _types(seed, n, fractions):
    """Op types by cumulative fractions of get, put, update (the rest: remove)."""
    get, put, update = fractions
    u = _uniform(seed, _TYPES, n)
    t = torch.full((n,), L.OP_REMOVE, dtype=torch.uint8, device="cuda")
    t[u < get + put + update] = L.OP_UPDATE
    t[u < get + put] = L.OP_PUT
    t[u < get] = L.OP_GET
    return t


def _by_type(types):
    """Order of a stable sort by op type: gets, puts, removes (a caller that
    collects its ops per type)."""
    return torch.sort(types, stable=True).indices


def _perm32(i):
    """A bijection on 32-bit numbers (as int64): distinct unstructured set keys."""
    m = 0xFFFFFFFF
    x = i & m
    x = ((x ^ (x >> 16)) * 0x7FEB352D) & m
    x = ((x ^ (x >> 15)) * 0x846CA68B) & m
    return x ^ (x >> 16)


def _set_keys(seed, index):
    """Set key number `index` of this seed (distinct for distinct numbers)."""
    k = _perm32(index + (seed * 0x9E3779B1 & 0xFFFFFFFF))
    return torch.where(k >> 31 > 0, k - (1 << 32), k).int()


def _packed(seed, n, median, what):
    """n values of lognormal length (clipped to 1..2048): packed bytes, offsets."""
    u1, u2 = _uniform(seed, what, n), _uniform(seed + 7919, what, n)
    z = torch.sqrt(-2.0 * torch.log1p(-u1)) * torch.cos(2.0 * math.pi * u2)
    size = torch.exp(math.log(median) + z).round().long().clamp_(1, 2048)
    off = torch.zeros(n + 1, dtype=torch.int64, device="cuda")
    off[1:] = torch.cumsum(size, 0)
    total = int(off[-1])
    data = _stream(seed, _BYTES + 16 * what, (total + 7) // 8).view(torch.uint8)[:total].clone()
    return data, off


def _zeros(*shape, dtype=torch.int64):
    return torch.zeros(shape, dtype=dtype, device="cuda")


# ----------------------------------------------------------------- prepare
def prepare(case, seed):
    return globals()["_prepare_" + case["kind"]](case, seed)


def _prepare_get(case, seed):
    m, items = _filled_map(case, seed)
    n = case["n"]
    keys = _at(seed, _KEYS, _ranks(seed, items, case["theta"], n))
    absent = _uniform(seed, _HITS, n) >= case["hit"]
    keys = torch.where(absent, _stream(seed, _NEW, n), keys)
    out = _zeros(n, 2) if case["width"] == 64 else _zeros(n)
    return {"kind": "get", "m": m, "keys": keys, "out": out, "width": case["width"]}


def _prepare_put(case, seed):
    m, items = _filled_map(case, seed)
    n, narrow = case["n"], case["width"] == 32
    keys = _at(seed, _KEYS, _ranks(seed, items, case["theta"], n))
    vals = _stream(seed, _VALUES, n)
    s = {"kind": "put", "m": m, "keys": keys, "vals": vals.int() if narrow else vals,
         "old": _zeros(n, dtype=torch.int32 if narrow else torch.int64), "width": case["width"]}
    run(s)  # from here on each pass finds the last pass's values
    return s


def _prepare_temporary(case, seed):
    m, _ = _filled_map(case, seed)
    n = case["n"]
    return {"kind": "temporary", "m": m, "keys": _stream(seed, _NEW, n),
            "vals": _stream(seed, _VALUES, n), "old": _zeros(n), "out": _zeros(n, 2)}


def _prepare_mixed(case, seed):
    m, items = _filled_map(case, seed)
    n = case["n"]
    types = _types(seed, n, (case["get"], case["put"], case["update"]))
    keys = _at(seed, _KEYS, _ranks(seed, items, case["theta"], n))
    vals = _stream(seed, _VALUES, n)
    if case["sorted"]:
        order = _by_type(types)
        types, keys, vals = types[order], keys[order], vals[order]
    if case["overlap"]:
        m.set_tuning(overlap=1)
    s = {"kind": "mixed", "m": m, "types": types, "keys": keys, "vals": vals,
         "out": _zeros(n, 2), "form": case["form"]}
    run(s)
    return s


def _queue_sizes(case):
    """Lognormal sizes (sigma 1.5) clipped to [1, 2^18], the same for every seed."""
    return W.lognormal_sizes(11, case["batches"], case["median"], 1.5, 1, 1 << 18)


def _prepare_queue(case, seed):
    m, items = _filled_map(case, seed)
    sizes = torch.from_numpy(_queue_sizes(case)).cuda()
    n = int(sizes.sum())
    types = _types(seed, n, (0.80, 0.15, 0.0))
    keys = _at(seed, _KEYS, _ranks(seed, items, case["theta"], n))
    vals = _stream(seed, _VALUES, n)
    # each batch lists its gets, then its puts, then its removes
    batch = torch.repeat_interleave(torch.arange(len(sizes), device="cuda"), sizes)
    order = torch.sort(batch * 4 + types.long(), stable=True).indices
    s = {"kind": "queue", "m": m, "types": types[order], "keys": keys[order],
         "vals": vals[order], "out": _zeros(n, 2)}
    m.execute_fused(s["types"], s["keys"], s["vals"], s["out"])
    s["graph"] = m.capture_fused(s["types"], s["keys"], s["vals"], s["out"])
    return s


def _prepare_set(case, seed):
    log2, n = case["log2"], case["n"]
    items = case["load"] << log2
    p = L.Set(log2, max(4096, (1 << log2) * max(1, case["load"] // 14) // 2 + 4096))
    for at in range(0, items, _CHUNK):
        p.insert(_set_keys(seed, torch.arange(at, min(items, at + _CHUNK), device="cuda")))
    new = torch.arange(items, items + 4 * n // 10, device="cuda")
    gone = max(1, n // 10)
    expired = torch.arange(gone, device="cuda") * (items // gone) + \
        _ranks(seed, items // gone, 0.0, gone)  # one of each equal share: distinct
    check = _ranks(seed, 2 * items, 0.0, n // 2, _HITS)  # half of them present
    k_new, k_old, k_check = (_set_keys(seed, x) for x in (new, expired, check))
    s = {"kind": "set", "p": p, "form": case["form"], "check": k_check, "new": k_new, "old": k_old}
    if case["form"] == "fused":
        # forward: check, add the new keys, drop the expired ones; back: the
        # same check, the expired keys return, the new ones leave
        def batch(put, drop):
            keys = torch.cat([k_check, put, drop])
            t = torch.cat([torch.full((len(k),), o, dtype=torch.uint8, device="cuda") for k, o in
                           ((k_check, L.OP_CONTAINS), (put, L.OP_INSERT), (drop, L.OP_REMOVE))])
            return t, keys, _zeros(len(keys), dtype=torch.bool)
        s["forward"], s["back"] = batch(k_new, k_old), batch(k_old, k_new)
    else:
        s["out"] = [_zeros(len(k), dtype=torch.bool)
                    for k in (k_check, k_new, k_old, k_check, k_old, k_new)]
    return s


def _prepare_kv(case, seed):
    keys = _stream(seed, _KEYS, case["keys"])
    first, first_off = _packed(seed, case["keys"], case["median"], _VALUES)
    puts = []
    for r in range(case["rounds"]):
        # distinct keys: each round overwrites its share of the store
        at = torch.randperm(case["keys"], device="cuda",
                            generator=torch.Generator("cuda").manual_seed(seed * 16 + r))
        data, off = _packed(seed + r + 1, case["puts"], case["median"], _VALUES)
        puts.append((keys[at[:case["puts"]]].contiguous(), data, off))
    heap = 4 * (first.numel() + sum(p[1].numel() for p in puts)) + (1 << 16)
    kv = L.KVStore(case["log2"], heap)
    kv.put(keys, first, first_off)
    n = case["reads"]
    s = {"kind": "kv", "kv": kv, "puts": puts, "reads": []}
    for r in range(case["rounds"]):
        k = _at(seed, _KEYS, _ranks(seed + r + 1, case["keys"] + case["keys"] // 16, 0.0, n))
        s["reads"].append({"keys": k, "len": _zeros(n, dtype=torch.int32), "off": _zeros(n),
                           "found": _zeros(n, dtype=torch.uint8),
                           "dst": _zeros(3 * n * case["median"] + 4096, dtype=torch.uint8)})
    run(s)  # the store is in the state that every later pass finds and leaves
    return s


def _prepare_serve(case, seed):
    m, items = _filled_map(case, seed)
    nreq = case["requests"]
    size = (_uniform(11, _SIZES, nreq) * case["max_ops"]).long() + 1  # the same for every seed
    total = int(size.sum())
    off = torch.zeros(nreq, dtype=torch.int64, device="cuda")
    off[1:] = torch.cumsum(size, 0)[:-1]
    keys = _at(seed, _KEYS, _ranks(seed, items, 0.99, total))
    types = (_uniform(seed, _TYPES, total) < 0.5).to(torch.uint8)
    vals = _stream(seed, _VALUES, total)
    host = [x.cpu().numpy() for x in (off, size.int(), types, keys, vals)]
    for i, kind in ((0, "u8"), (1, "u4"), (3, "u8"), (4, "u8")):
        host[i] = host[i].view(kind)
    sv = L.Server(m, arena_ops=1 << 20)
    zero = torch.zeros(nreq, dtype=torch.int64).numpy().view("u8")  # all due at once
    index = torch.arange(nreq, dtype=torch.int32).numpy().view("u4")
    torch.cuda.synchronize()  # the loop runs on a stream of its own
    s = {"kind": "serve", "sv": sv, "host": host, "arrival": zero, "index": index}
    run(s)  # from here on each pass finds the last pass's values
    return s


# --------------------------------------------------------------------- run
def run(s):
    return globals()["_run_" + s["kind"]](s)


def _run_get(s):
    if s["width"] == 64:
        s["m"].get(s["keys"], s["out"])
    else:
        L.lib().lsb_map_get_v32(s["m"].handle, s["keys"].data_ptr(), s["out"].data_ptr(),
                                s["keys"].numel(), torch.cuda.current_stream().cuda_stream)
    return s["out"]


def _run_put(s):
    if s["width"] == 64:
        s["m"].put(s["keys"], s["vals"], s["old"])
    else:
        L.lib().lsb_map_put_v32(s["m"].handle, s["keys"].data_ptr(), s["vals"].data_ptr(),
                                s["old"].data_ptr(), s["keys"].numel(),
                                torch.cuda.current_stream().cuda_stream)
    return s["old"]


def _run_temporary(s):
    s["m"].put(s["keys"], s["vals"], s["old"])
    s["m"].remove(s["keys"], s["out"])
    return s["old"], s["out"]


def _run_mixed(s):
    call = s["m"].execute_fused if s["form"] == "fused" else s["m"].execute
    call(s["types"], s["keys"], s["vals"], s["out"])
    return s["out"]


def _run_queue(s):
    s["graph"].launch()
    return s["out"]


def _run_set(s):
    p = s["p"]
    if s["form"] == "fused":
        for types, keys, out in (s["forward"], s["back"]):
            p.execute_fused(types, keys, out)
        return s["forward"][2], s["back"][2]
    out = s["out"]
    p.contains(s["check"], out[0])
    p.insert(s["new"], out[1])
    p.remove(s["old"], out[2])
    p.contains(s["check"], out[3])
    p.insert(s["old"], out[4])
    p.remove(s["new"], out[5])
    return out


def _run_kv(s):
    kv = s["kv"]
    totals = []
    for (keys, data, off), q in zip(s["puts"], s["reads"]):
        kv.put(keys, data, off)
        totals.append(kv.get(q["keys"], q["len"], q["off"], q["dst"], q["dst"].numel(), q["found"]))
    kv.compact()
    return [[q["len"], q["off"], q["found"], q["dst"]] for q in s["reads"]], totals


def _run_serve(s):
    sv, (off, size, types, keys, vals) = s["sv"], s["host"]
    sv.start()
    _, _, results = sv.run_load(s["arrival"], s["index"], off, size, types, keys, vals,
                                want_results=True)
    sv.stop()
    return results["found"], results["value"]


# -------------------------------------------------------------------- work
# Bytes of one op: its key, value and result, the 32-byte sector that holds the
# bucket's state and, for a key that is there, the sector that holds its slot.
# A write also stores its slot's sector; one that enters or leaves a key its
# state's sector too.
def work(case):
    return {"bytes": float(globals()["_bytes_" + case["kind"]](case)), "flops": 0.0}


def _bytes_get(case):
    result = 16 if case["width"] == 64 else 8
    return case["n"] * (8 + result + 32 + 32 * case["hit"])


def _bytes_put(case):
    return case["n"] * (8 + case["width"] // 4 + 32 + 2 * 32)


def _bytes_temporary(case):
    return case["n"] * ((24 + 32 + 64) + (24 + 64 + 64))


def _bytes_mixed(case):
    n, get = case["n"], case["get"]
    return n * (1 + 8 + 16 + 64) + n * (1 - get) * (8 + 32)


def _bytes_queue(case):
    n = int(_queue_sizes(case).sum())
    return n * (1 + 8 + 16 + 64) + n * 0.20 * (8 + 32)


def _bytes_set(case):
    n = case["n"]
    types = 1 if case["form"] == "fused" else 0
    reads = 2 * (n // 2) * (types + 4 + 1 + 48)
    return reads + 2 * (4 * n // 10 + n // 10) * (types + 4 + 1 + 64 + 32)


def _bytes_kv(case):
    mean = case["median"] * math.exp(0.5)  # of the lognormal lengths
    moved = case["puts"] * mean + case["reads"] * mean  # bytes in, bytes out
    ops = case["puts"] * (8 + 8 + 64 + 32) + case["reads"] * (8 + 4 + 8 + 1 + 64)
    return case["rounds"] * (2 * moved + ops) + case["keys"] * (2 * mean + 2 * 64)


def _bytes_serve(case):
    n = case["requests"] * (case["max_ops"] + 1) / 2
    return n * (17 + 16 + 64 + 0.5 * 32)


def exact(case, seed):
    """Results are stored words, found bits and bytes: nothing is computed."""
    return None
