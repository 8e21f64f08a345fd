"""The calls whose speed counts, as a program that uses the library makes them.

A case names an entry point (`op`) and its sizes:

  call     one column and one mask in device memory (`compressstore`), the drop-in call
  if       the selection is a comparison evaluated on the device (`compressstore_if`)
  pattern  the selection is periodic (`compressstore_pattern`)
  batch    a plan over many uneven columns, replayed as one graph (`Batch`)
  serve    a wave of requests through the serving loop (`Server`)

`prepare` puts payload, mask and an output of zeros in device memory, `run` makes the call, and
the outputs are the whole output buffers and the counts.
"""
import math
import random

import torch

import gpu_compressstore2_b200 as cs

DTYPES = {"u8": torch.uint8, "i16": torch.int16, "i32": torch.int32, "i64": torch.int64, "f32": torch.float32,
          "f64": torch.float64}
SECTOR = 32  # bytes of a payload line that can be left unread


def listed():
    return [
        # a filter over a whole resident column that keeps half of it: the library's headline call
        {"name": "call_f32_2p28_p50", "op": "call", "dtype": "f32", "n": 1 << 28, "mask": "iid", "p": 0.5},
        # a selective filter (a point lookup, an outlier search) over the same column
        {"name": "call_f32_2p28_p01", "op": "call", "dtype": "f32", "n": 1 << 28, "mask": "iid", "p": 0.01},
        # dropping the few bad rows of a 64-bit column (keys, timestamps); the planner knows the fraction
        {"name": "call_i64_ragged_p90", "op": "call", "dtype": "i64", "n": (1 << 27) - 77, "mask": "iid", "p": 0.9,
         "stated": 0.9},
        # a byte column (flags, dictionary codes) in storage order, where selected rows come in short runs
        {"name": "call_u8_2p29_runs8", "op": "call", "dtype": "u8", "n": 1 << 29, "mask": "runs", "p": 8.0},
        # a 16-bit column (codes, half-precision features) of a length that is no multiple of anything
        {"name": "call_i16_ragged_p50", "op": "call", "dtype": "i16", "n": (1 << 28) + 12345, "mask": "iid", "p": 0.5},
        # a vector of a vectorised engine: a small call, where latency and launches count
        {"name": "call_i32_2p20_p50", "op": "call", "dtype": "i32", "n": 1 << 20, "mask": "iid", "p": 0.5},
        # a row group of an ordinary table
        {"name": "call_i32_ragged_p10", "op": "call", "dtype": "i32", "n": (1 << 24) + 4099, "mask": "iid", "p": 0.1},
        # rows 96.. of a column, appended behind what earlier rows left in the output: the mask starts
        # inside a 16-byte group and the output at an arbitrary element
        {"name": "call_i32_rows_append", "op": "call", "dtype": "i32", "n": (1 << 26) - 1000, "mask": "iid", "p": 0.5,
         "in_off": 96, "mask_off": 3, "out_off": 5},
        # WHERE x > c without a mask in memory
        {"name": "if_f32_2p28_gt", "op": "if", "dtype": "f32", "n": 1 << 28, "cmp": ">", "p": 0.5},
        # every row of a fixed stride pattern (channels of interleaved samples)
        {"name": "pattern_i16_4of8", "op": "pattern", "dtype": "i16", "n": (1 << 28) + 5, "pattern": 0b10110010,
         "length": 8},
        # all columns of a table (uneven lengths, 4 and 8 bytes, any selectivity) in one plan
        {"name": "batch_256", "op": "batch", "columns": 256, "lo": 1 << 10, "hi": 1 << 24, "sizes": 1},
        # a burst of clients' requests over resident columns, from submission until the results were taken
        # out of the server's arena and their space given back
        {"name": "serve_32", "op": "serve", "columns": 32, "lo": 1 << 12, "hi": 1 << 24, "sizes": 2},
    ]


def _log_int(rng, lo, hi):
    return max(1, int(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choices(["call", "if", "pattern", "batch", "serve"], [12, 2, 2, 2, 1])[0]
    if op in ("batch", "serve"):
        top = rng.randrange(16, 25)
        return {"op": op, "columns": _log_int(rng, 4, 256 if op == "batch" else 32), "lo": 1 << rng.randrange(10, 13), "hi": 1 << top,
                "sizes": rng.randrange(1 << 30)}
    dtype = rng.choice(list(DTYPES)[:5] if op == "call" else list(DTYPES))
    w = DTYPES[dtype].itemsize
    if op == "pattern":
        dtype = rng.choice(["u8", "i16", "i32", "i64"])
        w = DTYPES[dtype].itemsize
        length = rng.randrange(1, 33)
        return {"op": op, "dtype": dtype, "n": _log_int(rng, 1 << 12, min(1 << 28, (1 << 30) // w)),
                "pattern": rng.randrange(1, 1 << length), "length": length}
    if op == "if":
        return {"op": op, "dtype": dtype, "n": _log_int(rng, 1 << 10, min(1 << 28, (1 << 30) // w)),
                "cmp": rng.choice(["<", "<=", ">", ">="]), "p": round(rng.uniform(0.005, 0.99), 3)}
    c = {"op": op, "dtype": dtype, "n": _log_int(rng, 1 << 10, min(1 << 29, (1 << 30) // w))}
    if rng.random() < 0.25:  # clustered selections, half of the rows selected
        c.update(mask="runs", p=round(math.exp(rng.uniform(math.log(4), math.log(4096))), 1))
    else:
        p = rng.choice([rng.uniform(0.05, 0.95), math.exp(rng.uniform(math.log(1e-3), math.log(0.05))),
                        1 - math.exp(rng.uniform(math.log(1e-3), math.log(0.05)))])
        c.update(mask="iid", p=round(p, 4))
        if rng.random() < 0.3:
            c["stated"] = c["p"]
    if rng.random() < 0.2:  # a part of a column, the output appended
        rows = 32 * rng.randrange(1, 64)
        c.update(n=min(c["n"], (1 << 28) // w), in_off=rows, mask_off=rows // 32, out_off=rng.randrange(1, 1000))
    return c


# ---------------------------------------------------------------- inputs
def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _payload(dtype, n, g):
    dt = DTYPES[dtype]
    if dt.is_floating_point:
        return torch.rand(n, dtype=dt, device="cuda", generator=g)
    words = (n * dt.itemsize + 7) // 8
    raw = torch.randint(-(1 << 63), (1 << 63) - 1, (words,), dtype=torch.int64, device="cuda", generator=g)
    return raw.view(dt)[:n]


def _selection(kind, p, n, g):
    """The selected rows as booleans: iid with probability p, or alternating runs of mean length p."""
    if kind == "iid":
        return torch.rand(n, device="cuda", generator=g) < p
    toggles = torch.rand(n, device="cuda", generator=g) < 1.0 / p
    return (torch.cumsum(toggles, 0, dtype=torch.int32) & 1).bool()


def _pack(sel):
    """LSB-first mask words (whole 16-byte groups) of the booleans."""
    n = sel.numel()
    padded = torch.zeros((n + 127) // 128 * 128, dtype=torch.uint8, device="cuda")
    padded[:n] = sel
    bits = padded.view(-1, 8)
    packed = bits[:, 0].clone()
    for b in range(1, 8):
        packed |= bits[:, b] << b
    return packed.view(torch.int32)


def _shifted(t, off):
    """t's values `off` elements past the start of an allocation."""
    if not off:
        return t
    room = torch.empty(t.numel() + off, dtype=t.dtype, device="cuda")
    room[off:] = t
    return room[off:]


def _columns(case):
    """(n, element bytes, p) of each column of a batch or of each request."""
    r = random.Random(case["sizes"])
    widths = [4, 8] if case["op"] == "batch" else [4]
    return [(_log_int(r, case["lo"], case["hi"]), r.choice(widths), r.uniform(0.01, 0.99))
            for _ in range(case["columns"])]


def _threshold(case):
    """The comparison's constant, for which a fraction p of uniform payloads is selected."""
    dt = DTYPES[case["dtype"]]
    at = case["p"] if case["cmp"] in ("<", "<=") else 1.0 - case["p"]
    if dt.is_floating_point:
        return at
    lo, hi = torch.iinfo(dt).min, torch.iinfo(dt).max
    return min(hi, lo + int(at * (float(hi) - float(lo))))


def _inputs(case, seed):
    """Payload and booleans of a call."""
    g = _generator(seed)
    return _payload(case["dtype"], case["n"], g), _selection(case["mask"], case["p"], case["n"], g)


def _table(case, seed):
    """Columns in device memory: (payload, mask words, n) each, every one 16-byte aligned."""
    g = _generator(seed)
    got = []
    for n, w, p in _columns(case):
        got.append((_payload("i32" if w == 4 else "i64", n, g), _pack(_selection("iid", p, n, g)), n))
    return got


def prepare(case, seed):
    op = case["op"]
    s = {"case": case, "count": torch.zeros(1, dtype=torch.int64, device="cuda")}
    if op == "call":
        x, sel = _inputs(case, seed)
        s["in"] = _shifted(x, case.get("in_off", 0))
        s["mask"] = _shifted(_pack(sel), case.get("mask_off", 0))
        s["whole"] = torch.zeros(case["n"] + case.get("out_off", 0), dtype=x.dtype, device="cuda")
        s["out"] = s["whole"][case.get("out_off", 0):]
    elif op in ("if", "pattern"):
        s["in"] = _payload(case["dtype"], case["n"], _generator(seed))
        s["whole"] = s["out"] = torch.zeros_like(s["in"])
        if op == "if":
            s["pred"] = cs.predicate(case["cmp"], _threshold(case), dtype=s["in"].dtype)
    elif op == "batch":
        table = _table(case, seed)
        s["table"] = table
        s["counts"] = torch.zeros(len(table), dtype=torch.int64, device="cuda")
        outs = {}
        for dt in (torch.int32, torch.int64):
            room = sum((n + 3) // 4 * 4 for x, _, n in table if x.dtype == dt)
            outs[dt] = [torch.zeros(room, dtype=dt, device="cuda"), 0]
        s["outs"] = [outs[torch.int32][0], outs[torch.int64][0]]
        columns = []
        for i, (x, mask, n) in enumerate(table):
            room, at = outs[x.dtype]
            columns.append((x, mask, room[at:at + n], n, s["counts"][i:i + 1]))
            outs[x.dtype][1] = at + (n + 3) // 4 * 4
        s["plan"] = cs.Batch(columns)
        side = torch.cuda.Stream()
        side.wait_stream(torch.cuda.current_stream())
        s["plan"].capture_graph(stream=side)
    else:
        s["table"] = _table(case, seed)
        room = sum(x.numel() * x.element_size() + 4096 for x, _, _ in s["table"])
        s["server"] = cs.Server(out_budget_bytes=max(room, 64 << 20))
        s["results"] = torch.zeros(sum(n for _, _, n in s["table"]), dtype=torch.int32, device="cuda")
        torch.cuda.synchronize()  # the server runs on streams of its own
    return s


def run(s):
    case = s["case"]
    op = case["op"]
    if op == "call":
        cs.compressstore(s["in"], s["mask"], s["out"], case["n"], s["count"], selectivity=case.get("stated", 0.0))
    elif op == "if":
        cs.compressstore_if(s["in"], s["out"], case["n"], s["pred"], s["count"])
    elif op == "pattern":
        cs.compressstore_pattern(s["in"], s["out"], case["n"], case["pattern"], case["length"], s["count"])
    elif op == "batch":
        s["plan"].run()
        return s["outs"] + [s["counts"]]
    else:
        server = s["server"]
        tickets = [server.submit(x, mask, n) for x, mask, n in s["table"]]
        done = [server.wait(t) for t in tickets]
        torch.cat([server.output(t, r) for t, r in zip(tickets, done)],
                  out=s["results"][:sum(r.count for r in done)])
        torch.cuda.current_stream().synchronize()  # before the space is given back
        for t in tickets:
            server.release(t)
        return [s["results"], torch.tensor([r.count for r in done])]
    return [s["whole"], s["count"]]


# ---------------------------------------------------------------- what a pass cannot do without
def _payload_bytes(n, w, kind, p):
    """Payload that has to be read: the 32-byte sectors that hold a selected row."""
    k = SECTOR // w
    untouched = (1.0 - p) ** k if kind == "iid" else 0.5 * (1.0 - 1.0 / p) ** (k - 1)
    return n * w * (1.0 - untouched)


def work(case):
    op = case["op"]
    if op in ("batch", "serve"):
        b = sum(_payload_bytes(n, w, "iid", p) + n / 8 + n * p * w for n, w, p in _columns(case))
        return {"bytes": b, "flops": 0}
    n, w = case["n"], DTYPES[case["dtype"]].itemsize
    if op == "call":
        share = case["p"] if case["mask"] == "iid" else 0.5
        return {"bytes": _payload_bytes(n, w, case["mask"], case["p"]) + n / 8 + n * share * w + 8, "flops": 0}
    if op == "if":  # every row is read, to be compared
        return {"bytes": n * w + n * case["p"] * w + 8, "flops": n}
    length, kept = case["length"], bin(case["pattern"]).count("1")
    k = SECTOR // w  # the sectors of one common period that hold a selected row
    period = length * k // math.gcd(length, k)
    touched = sum(any(case["pattern"] >> (i % length) & 1 for i in range(a, a + k)) for a in range(0, period, k))
    return {"bytes": n * w * touched * k / period + n * kept / length * w + 8, "flops": 0}


# ---------------------------------------------------------------- the same from plain torch
def exact(case, seed):
    """The outputs from torch's own indexing. Integer outputs are copies of their inputs' bits and are
    compared as they are."""
    op = case["op"]
    if op not in ("call", "if") or not DTYPES[case["dtype"]].is_floating_point:
        return None
    if op == "call":
        x, sel = _inputs(case, seed)
    else:
        x = _payload(case["dtype"], case["n"], _generator(seed))
        c = torch.tensor(_threshold(case), dtype=x.dtype, device="cuda")
        sel = {"<": x < c, "<=": x <= c, ">": x > c, ">=": x >= c}[case["cmp"]]
    kept = x[sel].double()
    whole = torch.zeros(case["n"] + case.get("out_off", 0), dtype=torch.float64, device="cuda")
    at = case.get("out_off", 0)
    whole[at:at + kept.numel()] = kept
    return [whole, torch.tensor([kept.numel()], device="cuda")]
