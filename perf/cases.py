"""What a user of this library has it do, as timed cases.

Every case goes through the public Python API (`Plan` and `Context` for
products that are resident on the device, `multiply` for the one-shot call on
host arrays, `Batch`, `Server`).  Operands are uniform random words with the
top bit of each operand set, the benchmark's own distribution.  Sizes are the
repository's: the plain workloads of `birdwing_b200/workloads.py`, the
2^12..2^20-bit batch mix and the serving mix, with ragged sizes between them.

A case is a dict of plain values; its `kind` says which form it takes:

  device    one product of device-resident operands (`Context.multiply_device`)
  oneshot   one product of host arrays (`multiply`: copies in and out)
  batch     `count` products of uneven sizes in one `Batch.run`, host arrays
  serve     `count` requests of mixed sizes submitted to a `Server`, waited for

All results are whole numbers, so they have one right value.
"""
import math
import random

import numpy as np
import torch

import birdwing_b200 as bw
from birdwing_b200 import workloads

AUTO, P32, P64 = bw.BW_PATH_AUTO, bw.BW_PATH_P32, bw.BW_PATH_P64


def _device(name, la, lb, path=AUTO, num_primes=0, square=False):
    return {"name": name, "kind": "device", "la": la, "lb": lb, "path": path,
            "num_primes": num_primes, "square": square}


def listed():
    return [
        # the smallest requests a server sees (2^10 bits): launches and latency
        _device("tiny_1kbit", 32, 24),
        # a ragged product of a few ten thousand bits
        _device("small_32kbit", 1000, 701),
        # the drop-in host call at the 2^20-bit workload, host arrays in and out
        {"name": "oneshot_1mbit", "kind": "oneshot", "la": 1 << 15, "lb": 1 << 15},
        # the plain 2^20-bit workload: 16-bit coefficients, three 30-bit primes
        _device("plain_1mbit", 1 << 15, 1 << 15, P32, 3),
        # ragged, unbalanced, some millions of bits, the library's own choice
        _device("ragged_8mbit", 270001, 180011),
        # 2^26-bit operands, the library's own choice
        _device("auto_64mbit", 1 << 21, 1 << 21),
        # ragged and unbalanced just under 2^28 bits, the library's own choice
        _device("auto_ragged_250mbit", 8000001, 7300003),
        # the benchmark's product: 2^28-bit operands on the 64-bit path
        _device("plain_256mbit", 1 << 23, 1 << 23, P64),
        # ... and its squaring
        _device("square_256mbit", 1 << 23, 1 << 23, P64, 0, True),
        # the huge product: 2^33-bit operands (1 GiB each), three passes
        _device("huge_8gbit", 1 << 28, 1 << 28, P64),
        # 4096 products of 2^12..2^20 bits, half on each path, host to host
        {"name": "batch_4096", "kind": "batch", "count": 4096, "lo": 12, "hi": 20},
        # a burst of mixed requests, squarings among them
        {"name": "serve_256", "kind": "serve", "count": 256, "lo": 10, "hi": 20},
    ]


def _log_int(rng, lo, hi):
    """An integer in [lo, hi], uniform over its logarithm."""
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng: random.Random):
    kind = rng.choice(["device"] * 7 + ["oneshot", "batch", "serve"])
    if kind == "device":
        c = _device("", 0, 0)
        del c["name"]
        c["la"] = _log_int(rng, 16, 1 << 23)
        c["square"] = rng.random() < 0.2
        # the second operand is 1/8 to 1 of the first
        c["lb"] = c["la"] if c["square"] else max(1, int(c["la"] * 2.0 ** rng.uniform(-3, 0)))
        c["path"] = rng.choice([AUTO, AUTO, P64])
        if c["path"] == AUTO and c["la"] <= 1 << 20 and rng.random() < 0.3:
            c["path"], c["num_primes"] = P32, rng.choice([2, 3])
        return c
    if kind == "oneshot":
        la = _log_int(rng, 64, 1 << 20)
        return {"kind": kind, "la": la, "lb": max(1, int(la * 2.0 ** rng.uniform(-3, 0)))}
    lo = rng.randrange(10, 16)
    return {"kind": kind, "count": _log_int(rng, 16, 2048 if kind == "batch" else 256),
            "lo": lo, "hi": rng.randrange(lo + 1, 21)}


def _device_words(n, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    x = torch.randint(-(1 << 31), 1 << 31, (n,), dtype=torch.int32, device="cuda", generator=g)
    x[-1:].bitwise_or_(-(1 << 31))
    return x


def _mix(case, seed):
    """The operands of a batch or of a burst of requests, and one output array
    with a slice of it for each product."""
    rng = np.random.default_rng([seed, 77])
    items = []
    if case["kind"] == "batch":
        for path, la, lb in workloads.batch_sizes(case["count"], 3, case["lo"], case["hi"]):
            items.append((path, workloads.rand_operand(rng, la), workloads.rand_operand(rng, lb)))
    else:
        for la, lb, sq in workloads.serving_sizes(case["count"], 5, case["lo"], case["hi"]):
            a = workloads.rand_operand(rng, la)
            items.append((AUTO, a, a if sq else workloads.rand_operand(rng, lb)))
    out = np.zeros(sum(a.size + b.size for _, a, b in items), dtype=np.uint32)
    parts, at = [], 0
    for _, a, b in items:
        parts.append(out[at: at + a.size + b.size])
        at += a.size + b.size
    return items, out, parts


def _host_pair(case, seed):
    rng = np.random.default_rng([seed, 78])
    return (workloads.rand_operand(rng, case["la"]), workloads.rand_operand(rng, case["lb"]))


def _device_pair(case, seed):
    a = _device_words(case["la"], 2 * seed)
    return a, a if case["square"] else _device_words(case["lb"], 2 * seed + 1)


def prepare(case, seed):
    s = dict(case)
    if case["kind"] == "device":
        s["a"], s["b"] = _device_pair(case, seed)
        s["out"] = torch.empty(case["la"] + case["lb"], dtype=torch.int32, device="cuda")
        s["plan"] = bw.Plan(case["la"], case["lb"], case["path"], case["num_primes"])
        s["ctx"] = bw.Context(s["plan"])
        # the context's stream is its own: the operands have to be there
        torch.cuda.synchronize()
    elif case["kind"] == "oneshot":
        s["a"], s["b"] = _host_pair(case, seed)
    else:
        items, s["out"], parts = _mix(case, seed)
        s["items"], s["parts"] = items, parts
        if case["kind"] == "batch":
            s["batch"] = bw.Batch()
            for (path, a, b), o in zip(items, parts):
                s["batch"].add(a, b, o, path)
        else:
            s["server"] = bw.Server()
            s["server"].prewarm(17)
    return s


def run(s):
    if s["kind"] == "device":
        a, b, out = s["a"], s["b"], s["out"]
        s["ctx"].multiply_device(a.data_ptr(), s["la"], b.data_ptr(), s["lb"], out.data_ptr(),
                                 out.numel())
        return out
    if s["kind"] == "oneshot":
        return bw.multiply(s["a"], s["b"]).view(np.int32)
    if s["kind"] == "batch":
        s["batch"].run()
        return s["out"].view(np.int32)
    srv = s["server"]
    tickets = [srv.submit(a, b, o) for (_, a, b), o in zip(s["items"], s["parts"])]
    for t in tickets:
        srv.wait(t)
    return s["out"].view(np.int32)


def work(case):
    """Operands read once, the product written once.  The arithmetic between
    them is on whole numbers: no floating-point operation is one that the path
    cannot do without."""
    if case["kind"] in ("device", "oneshot"):
        la, lb = case["la"], case["lb"]
        words = la + (0 if case.get("square") else lb) + la + lb
    elif case["kind"] == "batch":
        words = sum(2 * (la + lb) for _, la, lb in
                    workloads.batch_sizes(case["count"], 3, case["lo"], case["hi"]))
    else:
        words = sum(2 * (la + lb) - (lb if sq else 0) for la, lb, sq in
                    workloads.serving_sizes(case["count"], 5, case["lo"], case["hi"]))
    return {"bytes": 4.0 * words, "flops": 0.0}


def _product(a, b):
    n = 4 * (a.size + b.size)
    p = int.from_bytes(a.tobytes(), "little") * int.from_bytes(b.tobytes(), "little")
    return np.frombuffer(p.to_bytes(n, "little"), dtype=np.int32).copy()


def exact(case, seed):
    """The products by Python's integers, where those take seconds at most."""
    if case["kind"] in ("device", "oneshot"):
        if max(case["la"], case["lb"]) > 1 << 19:
            return None
        if case["kind"] == "oneshot":
            return _product(*_host_pair(case, seed))
        a, b = _device_pair(case, seed)
        return torch.from_numpy(_product(a.cpu().numpy(), b.cpu().numpy()))
    items, _, _ = _mix(case, seed)
    return np.concatenate([_product(a, b) for _, a, b in items])
