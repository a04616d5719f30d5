"""The workloads the sort's speed is followed on.

Each case is one call (or one round of requests) that a program using
b200sort makes: packed batches of equal-length arrays through the C ABI
binding and the PyTorch operators, ragged CSR batches through a plan and the
PyTorch operator, single long arrays, arrays of one thread-block cluster each,
and requests to the continuous-batching server.

A case is a dict:
  kind    "packed" (b200sort.sort_packed into the caller's buffer),
          "packed_op" / "ragged_op" (torch.ops.b200sort.*, a new output),
          "ragged" (a plan the program keeps), "serve" (server requests)
  elem    "i32", "i32_i32", "u64" or "u64_i32" (see b200sort.DTYPES)
  stable  ties in input order (records)
  arrays  arrays of the batch, or requests of the round
  n       their length (packed), or the longest one (ragged, serve)
  lo      the shortest one (ragged, serve): lengths are spread over [lo, n],
          uniform in their logarithm, in an order that the seed gives
  keys    "uniform" over the full key range, "distinct16" (16 values), or
          "swap8" (sorted, then elements exchanged at most 8 places apart)

Record payloads are the record's position in the batch, as the reference's
generator sets them.
"""
import math
import os
import sys

import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PKG = os.path.join(ROOT, "cuda-sort_b200")
if PKG not in sys.path:
    sys.path.insert(0, PKG)

import b200sort as bs  # noqa: E402
import b200sort_torch  # noqa: E402,F401  (registers torch.ops.b200sort)

BYTES = {"i32": 4, "i32_i32": 8, "u64": 8, "u64_i32": 16}
MAX_LENGTH = {"i32": 131072, "i32_i32": 65536, "u64": 65536, "u64_i32": 65536}


def _case(kind, elem, arrays, n, lo=0, stable=False, keys="uniform", name=None):
    c = {"kind": kind, "elem": elem, "stable": stable, "arrays": arrays, "n": n, "lo": lo, "keys": keys}
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # the benchmark's headline: one batch of 4096 short key arrays
        _case("packed", "i32", 4096, 1024, name="keys_4096x1024"),
        # very many very short record arrays (neighbour lists, top-k candidates)
        _case("packed", "i32_i32", 131072, 32, name="records_131072x32"),
        # an odd length just above a power of two, with heavy ties
        _case("packed", "i32_i32", 32513, 129, keys="distinct16", name="records_32513x129_ties"),
        # a length that is no power of two, one warp per array
        _case("packed", "i32_i32", 4194, 1000, name="records_4194x1000"),
        # 64-bit keys (hashes, packed coordinates) from PyTorch
        _case("packed_op", "u64", 2097, 2000, name="u64_op_2097x2000"),
        # records with ties kept in input order, nearly sorted input
        _case("packed", "i32_i32", 1398, 3000, stable=True, keys="swap8", name="stable_records_1398x3000"),
        # the smallest call: one short array, where the launch is what counts
        _case("packed", "i32_i32", 1, 300, name="one_array_300"),
        # one long array alone on the GPU
        _case("packed", "i32_i32", 1, 30000, name="one_array_30000"),
        # the ragged batch of the benchmark, through a plan kept by the program
        _case("ragged", "i32_i32", 200000, 8192, lo=1, name="ragged_200000"),
        # a modest ragged batch of key arrays from PyTorch
        _case("ragged_op", "i32", 1000, 8192, lo=1, name="ragged_op_keys_1000"),
        # arrays longer than one CTA holds
        _case("packed", "i32_i32", 256, 65536, name="records_256x65536"),
        # a burst of requests of very different sizes to the server
        _case("serve", "i32_i32", 256, 65536, lo=16, name="serve_256"),
    ]


def _log_int(rng, lo, hi):
    return min(hi, max(lo, int(math.exp(rng.uniform(math.log(lo), math.log(hi + 1))))))


def draw(rng):
    kind = rng.choice(["packed", "packed", "packed", "packed_op", "ragged", "ragged_op", "serve"])
    keys = rng.choice(["uniform", "uniform", "distinct16", "swap8"] if kind.startswith("packed")
                      else ["uniform", "uniform", "distinct16"])
    if kind.startswith("packed"):
        elem, stable = rng.choice([("i32", False), ("i32_i32", False), ("i32_i32", False), ("i32_i32", True),
                                   ("u64", False), ("u64_i32", False), ("u64_i32", True)])
        n = _log_int(rng, 8, MAX_LENGTH[elem])
        total = _log_int(rng, n, 1 << 22) if n < (1 << 22) else n
        return _case(kind, elem, max(1, total // n), n, stable=stable, keys=keys)
    if kind == "serve":
        return _case(kind, "i32_i32", _log_int(rng, 1, 256), _log_int(rng, 1024, 65536), lo=16, keys=keys)
    elem, stable = rng.choice([("i32", False), ("i32_i32", False), ("i32_i32", True), ("u64", False)])
    return _case(kind, elem, _log_int(rng, 4, 20000), _log_int(rng, 64, 8192), lo=1, stable=stable, keys=keys)


def _keys(case, total, gen):
    """int32 or int64 keys (the bit patterns of the unsigned ones), flat."""
    wide = case["elem"].startswith("u64")
    dt = torch.int64 if wide else torch.int32

    def uniform(count):
        words = torch.randint(-2 ** 31, 2 ** 31, (count * (2 if wide else 1),), generator=gen, device="cuda",
                              dtype=torch.int64).to(torch.int32)
        return words.view(dt)

    if case["keys"] == "distinct16":
        values = uniform(16)
        return values[torch.randint(0, 16, (total,), generator=gen, device="cuda")]
    keys = uniform(total)
    if case["keys"] == "swap8":
        flip = torch.iinfo(dt).min if wide else 0  # unsigned order of 64-bit patterns
        rows = (keys.view(-1, case["n"]) ^ flip).sort(dim=1).values ^ flip
        width = case["n"] // 16 * 16
        if width:
            body = rows[:, :width].reshape(-1, 16)
            i = torch.randint(0, 8, (body.shape[0], 1), generator=gen, device="cuda")
            j = i + torch.randint(1, 9, (body.shape[0], 1), generator=gen, device="cuda")
            a, b = body.gather(1, i), body.gather(1, j)
            body = body.scatter(1, i, b).scatter(1, j, a)
            rows[:, :width] = body.reshape(-1, width)
        keys = rows.reshape(-1).contiguous()
    return keys


def _elements(case, total, gen):
    keys = _keys(case, total, gen)
    if case["elem"] in ("i32", "u64"):
        return keys
    place = torch.arange(total, device="cuda", dtype=torch.int32)
    if case["elem"] == "i32_i32":
        return torch.stack([keys, place], dim=1).contiguous()
    out = torch.zeros((total, 4), device="cuda", dtype=torch.int32)
    out[:, :2] = keys.view(torch.int32).view(-1, 2)
    out[:, 2] = place
    return out


def _lengths(case):
    """The batch's lengths, shortest first: the middles of equal steps of the logarithm."""
    u = (torch.arange(case["arrays"], device="cuda", dtype=torch.float64) + 0.5) / case["arrays"]
    lo, hi = math.log(case["lo"]), math.log(case["n"])
    return torch.exp(lo + u * (hi - lo)).floor().to(torch.int64).clamp(case["lo"], case["n"])


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    dtype = bs.DTYPES[case["elem"]]
    flags = bs.STABLE if case["stable"] else 0
    state = {"case": case, "dtype": dtype, "flags": flags}
    if case["kind"].startswith("packed"):
        state["values"] = _elements(case, case["arrays"] * case["n"], gen)
        if case["kind"] == "packed":
            state["out"] = torch.empty_like(state["values"])
        return state
    offsets = torch.zeros(case["arrays"] + 1, device="cuda", dtype=torch.int64)
    order = torch.randperm(case["arrays"], generator=gen, device="cuda")
    offsets[1:] = torch.cumsum(_lengths(case)[order], 0)
    total = int(offsets[-1].item())
    state["values"] = _elements(case, total, gen)
    state["offsets"] = offsets.to(torch.int32)
    if case["kind"] == "ragged_op":
        return state
    state["out"] = torch.empty_like(state["values"])
    if case["kind"] == "ragged":
        state["plan"] = bs.Plan(dtype, case["arrays"], flags, torch.cuda.current_device())
        return state
    host = offsets.tolist()
    size = BYTES[case["elem"]]
    src, dst = state["values"].data_ptr(), state["out"].data_ptr()
    state["requests"] = [(src + a * size, dst + a * size, b - a) for a, b in zip(host, host[1:])]
    state["server"] = bs.Server(dtype, budget_bytes=256 << 20, flags=flags, device=torch.cuda.current_device())
    torch.cuda.synchronize()  # the server reads the inputs on streams of its own
    return state


def run(state):
    case, values = state["case"], state["values"]
    kind = case["kind"]
    if kind == "packed_op":
        return torch.ops.b200sort.sort_packed(values, case["n"], case["stable"])
    if kind == "ragged_op":
        return torch.ops.b200sort.sort_ragged(values, state["offsets"], case["stable"])
    out = state["out"]
    if kind == "serve":
        server = state["server"]
        for src, dst, n in state["requests"]:
            server.submit(src, dst, n)
        server.drain()
        return out
    stream = torch.cuda.current_stream().cuda_stream
    if kind == "ragged":
        state["plan"].sort(values.data_ptr(), out.data_ptr(), state["offsets"].data_ptr(), case["arrays"], stream)
    else:
        bs.sort_packed(state["dtype"], values.data_ptr(), out.data_ptr(), case["n"], case["arrays"], state["flags"],
                       None, stream)
    return out


def work(case):
    size = BYTES[case["elem"]]
    if case["kind"].startswith("packed"):
        return {"bytes": 2 * size * case["arrays"] * case["n"], "flops": 0}
    lo, hi = case["lo"], case["n"]
    mean = (hi - lo) / math.log(hi / lo) if hi > lo else lo  # of the log-uniform lengths
    return {"bytes": case["arrays"] * (2 * size * mean + 4), "flops": 0}


def exact(case, seed):
    """Keys alone have one sorted order, and stable records too; the order of
    equal keys in the default mode is the reference network's and has no plain
    statement."""
    if not (case["elem"] in ("i32", "u64") or case["stable"]) or not case["kind"].startswith("packed"):
        return None
    gen = torch.Generator(device="cuda").manual_seed(seed)
    values = _elements(case, case["arrays"] * case["n"], gen)
    shape = (case["arrays"], case["n"])
    if case["elem"].startswith("u64"):
        keys = values.view(torch.int64) if case["elem"] == "u64" else values[:, :2].contiguous().view(torch.int64)
        keys = keys.reshape(shape) ^ torch.iinfo(torch.int64).min
    else:
        keys = values.reshape(*shape, -1)[:, :, 0].to(torch.int64)
    order = keys.sort(dim=1, stable=True).indices
    order = (order + torch.arange(case["arrays"], device="cuda").view(-1, 1) * case["n"]).reshape(-1)
    return values[order]
