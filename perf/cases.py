"""The work whose speed is followed: device and host sorts, key + item sorts, top-k, selection and
batched sorts, from the smallest calls to the largest, through the entry points a program calls.

Keys lie in torch tensors on the GPU (unsigned keys as the signed tensor of the same bits, with the
key type passed along).  The sorts are in place, so a pass first refills its working buffer from
the unsorted input, as a program that sorts one buffer again and again does.
"""
import math

import numpy as np
import torch

from hpcsharp_b200 import algorithm, native, workloads

# key type -> (tensor type, key bytes)
TYPES = {
    "u32": (torch.int32, 4),
    "i32": (torch.int32, 4),
    "f32": (torch.float32, 4),
    "u64": (torch.int64, 8),
    "i64": (torch.int64, 8),
    "f64": (torch.float64, 8),
}


def listed():
    return [
        # the smallest calls: a thousand keys, where launches and latency are the whole time
        {"name": "sort_u32_1k", "kind": "sort", "dtype": "u32", "dist": "uniform", "n": 1_000},
        # a column or an index of a hundred thousand small signed values, an odd length
        {"name": "sort_i32_100k", "kind": "sort", "dtype": "i32", "dist": "normal", "n": 100_003},
        # sorting a million rows by a 32-bit key: key + row index
        {"name": "pairs_u32_1m", "kind": "pairs", "dtype": "u32", "dist": "uniform", "n": 1_000_003},
        # the extension method on an ordinary host array: copies in and out included
        {"name": "host_i32_1m", "kind": "host", "dtype": "i32", "dist": "normal", "n": 1_000_003},
        # the benchmark's ordinary array: ten million keys, which stay in the L2 cache
        {"name": "sort_u32_10m", "kind": "sort", "dtype": "u32", "dist": "uniform", "n": 10_000_000},
        # in-place selection around the median of a large float array
        {"name": "select_f32_33m", "kind": "select", "dtype": "f32", "dist": "normal", "n": 33_554_467, "k": 16_777_233},
        # the thousand largest of a very large array
        {"name": "topk_u32_256m", "kind": "topk", "dtype": "u32", "dist": "uniform", "n": 1 << 28, "k": 1_000},
        # large float keys: normal values crowd a few sign and exponent bytes
        {"name": "sort_f32_67m", "kind": "sort", "dtype": "f32", "dist": "normal", "n": 67_108_879},
        # large 64-bit keys, a ragged length
        {"name": "sort_u64_50m", "kind": "sort", "dtype": "u64", "dist": "uniform", "n": 50_000_017},
        # Zipf-distributed 64-bit keys (few identifiers hold most rows) with a row index
        {"name": "pairs_u64_zipf_50m", "kind": "pairs", "dtype": "u64", "dist": "zipf", "n": 50_000_000},
        # thousands of arrays of mixed length and type in one planned call
        {"name": "batch_16k_arrays", "kind": "batch", "arrays": 16_384, "keys": 62_500_000},
        # the headline: 2^28 uniform keys
        {"name": "sort_u32_256m", "kind": "sort", "dtype": "u32", "dist": "uniform", "n": 1 << 28},
    ]


def _log_size(rng, lo, hi):
    return int(math.exp(rng.uniform(math.log(lo), math.log(hi))))


def draw(rng):
    kind = rng.choice(["sort", "sort", "sort", "sort", "pairs", "pairs", "topk", "select", "batch", "host"])
    if kind == "batch":
        arrays = _log_size(rng, 1_024, 16_384)
        return {"kind": kind, "arrays": arrays, "keys": arrays * rng.randrange(1_000, 3_815)}
    if kind == "host":
        return {"kind": kind, "dtype": rng.choice(["u32", "i32"]), "dist": "uniform", "n": _log_size(rng, 10_000, 4_000_000)}
    dtype = rng.choice(["u32", "i32", "f32", "u64", "i64", "f64"])
    dist = {"u32": ["uniform"], "i32": ["normal", "uniform"], "f32": ["normal"], "u64": ["uniform", "and3", "zipf"],
            "i64": ["uniform"], "f64": ["normal"]}[dtype]
    case = {"kind": kind, "dtype": dtype, "dist": rng.choice(dist)}
    most = 1 << 28 if TYPES[dtype][1] == 4 else 1 << 26
    if kind == "pairs":
        case["n"] = _log_size(rng, 10_000, min(most // 2, 1 << 26))
    elif kind == "sort":
        case["n"] = _log_size(rng, 1_000, most)
    else:
        n = case["n"] = _log_size(rng, 100_000, most)
        case["k"] = _log_size(rng, 10, min(100_000, n // 2)) if kind == "topk" else rng.randrange(n)
    return case


def _keys(case, dtype, n, gen):
    """n keys of `dtype` on the GPU, of the case's distribution."""
    dev = torch.device("cuda", 0)
    dist = case.get("dist", "normal" if dtype in ("i32", "f32", "f64") else "uniform")
    if dtype in ("f32", "f64"):
        return torch.randn(n, dtype=TYPES[dtype][0], device=dev, generator=gen)
    if dist == "normal":  # signed values of deviation 2^20
        return torch.randn(n, device=dev, generator=gen).mul_(float(1 << 20)).round_().to(TYPES[dtype][0])
    if dist == "zipf":  # a million identifiers spread over 64 bits, their ranks by exponent 1.1
        u = torch.rand(n, dtype=torch.float64, device=dev, generator=gen)
        return u.mul_(1e6 ** -0.1 - 1.0).add_(1.0).pow_(-10.0).to(torch.int64).mul_(-7046029254386353131)

    def uniform():
        lo, hi = (-(1 << 31), 1 << 31) if TYPES[dtype][1] == 4 else (-(1 << 63), (1 << 63) - 1)
        return torch.randint(lo, hi, (n,), dtype=TYPES[dtype][0], device=dev, generator=gen)

    if dist == "and3":  # sparse bits: the AND of three uniform keys
        return uniform() & uniform() & uniform()
    return uniform()


def prepare(case, seed):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(int(seed))
    state = {"case": case, "ctx": native.default_context()}
    if case["kind"] == "batch":
        _, state["src"], state["work"], segments = _batch(case, gen)
        state["plan"] = state["ctx"].segplan(segments)
        return state
    keys = _keys(case, case["dtype"], case["n"], gen)
    if case["kind"] == "host":
        state["src"] = keys.cpu().numpy().view(native.NP_OF[case["dtype"]])
        state["work"] = np.empty_like(state["src"])
        return state
    state["src"] = keys
    if case["kind"] == "topk":
        state["out"] = torch.empty(case["k"], dtype=keys.dtype, device=keys.device)
    else:
        state["work"] = torch.empty_like(keys)
    if case["kind"] == "pairs":
        state["rows"] = torch.arange(case["n"], dtype=torch.int32, device=keys.device)
        state["items"] = torch.empty_like(state["rows"])
    return state


def _batch(case, gen):
    """One pool of keys per type, every array on a 16-byte boundary; the arrays as segments."""
    lengths, dtypes = workloads.batched_lengths(count=case["arrays"], target_total=case["keys"])
    layout, size = [], {}
    for n, dt in zip(lengths, dtypes):
        step = workloads.ALIGN_BYTES // TYPES[dt][1]
        at = size.get(dt, 0)
        layout.append((dt, at, int(n)))
        size[dt] = at + (int(n) + step - 1) // step * step
    src = {dt: _keys({}, dt, size[dt], gen) for dt in sorted(size)}
    work = {dt: torch.empty_like(src[dt]) for dt in src}
    segments = [((work[dt].data_ptr() + at * TYPES[dt][1], n), dt) for dt, at, n in layout]
    return layout, src, work, segments


def run(state):
    case, ctx = state["case"], state["ctx"]
    kind = case["kind"]
    if kind == "host":
        np.copyto(state["work"], state["src"])
        return algorithm.SortRadixPar(state["work"])
    stream = native.torch_stream()
    if kind == "batch":
        for dt, pool in state["work"].items():
            pool.copy_(state["src"][dt])
        state["plan"].execute(stream=stream)
        return state["work"]
    if kind == "topk":
        ctx.topk_largest_dev(state["src"], case["k"], state["out"], dtype=case["dtype"], stream=stream)
        return state["out"]
    state["work"].copy_(state["src"])
    if kind == "select":
        ctx.select_topk_dev(state["work"], case["k"], dtype=case["dtype"], stream=stream)
    elif kind == "pairs":
        state["items"].copy_(state["rows"])
        ctx.sort_pairs_dev(state["work"], state["items"], dtype=case["dtype"], stream=stream)
        return state["work"], state["items"]
    else:
        ctx.sort_dev(state["work"], dtype=case["dtype"], stream=stream)
    return state["work"]


def work(case):
    if case["kind"] == "batch":
        # four key types, drawn evenly: three of 4 bytes and one of 8
        return {"bytes": 2.0 * case["keys"] * 5, "flops": 0}
    n, w = case["n"], TYPES[case["dtype"]][1]
    if case["kind"] == "topk":
        return {"bytes": float((n + case["k"]) * w), "flops": 0}
    if case["kind"] == "pairs":
        return {"bytes": 2.0 * n * (w + 4), "flops": 0}
    return {"bytes": 2.0 * n * w, "flops": 0}


def _signed(keys, dtype):
    """Unsigned bits as signed values of the same order (and back)."""
    if dtype == "u32":
        return keys ^ -(1 << 31)
    if dtype == "u64":
        return keys ^ -(1 << 63)
    return keys


def exact(case, seed):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(int(seed))
    if case["kind"] == "batch":
        layout, src, _, _ = _batch(case, gen)
        out = {}
        for dt, pool in src.items():
            # array i's keys belong to group 2 i, the gap behind it (left as it is) to group 2 i + 1
            group = torch.zeros(pool.numel() + 1, dtype=torch.int64)
            for d, at, n in layout:
                if d == dt:
                    group[at] += 1
                    group[at + n] += 1
            group = torch.cumsum(group[:-1], 0).to(pool.device)
            at = torch.arange(pool.numel(), device=pool.device)
            _, by_key = torch.sort(_signed(pool, dt), stable=True)
            gap = _gaps(layout, dt, pool.numel()).to(pool.device)
            _, by_group = torch.sort(group[by_key], stable=True)
            got = pool[by_key[by_group]]
            out[dt] = torch.where(gap, pool, got) if bool(gap.any()) else got
            del at
        return out
    dt = case["dtype"]
    keys = _keys(case, dt, case["n"], gen)
    if case["kind"] == "pairs":
        got, rows = torch.sort(_signed(keys, dt), stable=True)
        return _signed(got, dt), rows.to(torch.int32)
    if case["kind"] == "select":
        x = _signed(keys, dt)
        v = torch.sort(x).values[case["k"]]
        return torch.cat([keys[x < v], keys[x == v], keys[x > v]])
    got = _signed(torch.sort(_signed(keys, dt)).values, dt)
    if case["kind"] == "topk":
        return got[case["n"] - case["k"]:]
    if case["kind"] == "host":
        return got.cpu().numpy().view(native.NP_OF[dt])
    return got


def _gaps(layout, dtype, size):
    gap = torch.ones(size, dtype=torch.bool)
    for d, at, n in layout:
        if d == dtype:
            gap[at:at + n] = False
    return gap
