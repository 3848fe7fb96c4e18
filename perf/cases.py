"""The sort engine's performance cases: the work its users have it do, called through the public Python binding.

Every case is device-resident unless it says otherwise: the caller holds the keys on the GPU, keeps its
unsorted copy, and sorts a work buffer in place on its own stream with scratch it allocated once. A pass of an
in-place entry point therefore copies the keys into the work buffer and sorts them there. The engine only
moves keys and values, it computes none, so results are returned as raw bits (integers of the key's width).
"""
import importlib.util
import math
import os
import sys

import numpy as np
import torch

WIDTH = {"u32": 4, "i32": 4, "f32": 4, "u64": 8, "i64": 8, "f64": 8}
DISTS = ("uniform", "normal", "zipf", "few", "nearly")

_shared = {}


def _mgs():
    if "mgs" in sys.modules:
        return sys.modules["mgs"]
    path = os.path.join(os.getcwd(), "multi-gpu-sorting_b200", "mgs.py")
    spec = importlib.util.spec_from_file_location("mgs", path)
    mod = importlib.util.module_from_spec(spec)
    sys.modules["mgs"] = mod
    spec.loader.exec_module(mod)
    return mod


def _engine():
    """The program's one engine context and the stream it sorts on."""
    if not _shared:
        _shared["ctx"] = _mgs().Context(0)
        _shared["stream"] = torch.cuda.Stream()
    return _shared["ctx"], _shared["stream"]


def listed():
    return [
        # The smallest calls: a few hundred rows of a query result. Latency and launches are all of it.
        {"name": "sort_u32_1k", "op": "sort", "dtype": "u32", "n": 1000, "dist": "uniform"},
        # A small float column with -0.0 and NaN among its values, ragged size.
        {"name": "sort_f32_50k", "op": "sort", "dtype": "f32", "n": 50_021, "dist": "normal"},
        # 8-byte ids with many duplicates: one partition of a join or a deduplication.
        {"name": "sort_i64_1m", "op": "sort", "dtype": "i64", "n": 1 << 20, "dist": "few"},
        # A skewed integer column (Zipf-distributed values, odd size) of ordinary size.
        {"name": "sort_u32_16m_zipf", "op": "sort", "dtype": "u32", "n": (1 << 24) + 13, "dist": "zipf"},
        # Doubles at an ordinary large size, ragged.
        {"name": "sort_f64_100m", "op": "sort", "dtype": "f64", "n": 100_000_003, "dist": "normal"},
        # The headline benchmark's keys: 2^30 uniform uint32.
        {"name": "sort_u32_1g", "op": "sort", "dtype": "u32", "n": 1 << 30, "dist": "uniform"},
        # Key-value sort: 4-byte keys with row ids.
        {"name": "pairs_u32_u32_16m", "op": "pairs", "dtype": "u32", "n": 1 << 24, "dist": "uniform", "value_bytes": 4},
        # Ranking by score: floats descending, with their indices.
        {"name": "rank_f32_desc_200k", "op": "range", "dtype": "f32", "n": 200_003, "dist": "normal",
         "value_bytes": 4, "begin": 0, "end": 32, "descending": True},
        # A batch of 10^5 segments of Zipf-distributed lengths (the batched workload of the benchmark).
        {"name": "segmented_u32_100k", "op": "segmented", "dtype": "u32", "n": 1 << 28, "dist": "uniform",
         "segments": 100_000, "lengths": "zipf"},
        # A small batch that is sorted again and again: 1024 segments in a recorded plan, replayed per batch.
        {"name": "plan_segments_1k", "op": "plan", "dtype": "u32", "n": 1 << 18, "dist": "uniform",
         "segments": 1024, "lengths": "even"},
        # Merging the sorted runs of an earlier phase.
        {"name": "kway_u32_k16", "op": "kway", "dtype": "u32", "n": 1 << 28, "dist": "uniform", "runs": 16},
        # TanasicSort on one GPU: keys in pinned host memory, copied in, sorted and copied back.
        {"name": "host_u32_32m", "op": "host", "dtype": "u32", "n": 1 << 25, "dist": "uniform"},
    ]


def _log_size(rng, lo_bits, hi_bits):
    """A size spread over the logarithm of [2^lo, 2^hi], odd ones among them."""
    n = int(2.0 ** rng.uniform(lo_bits, hi_bits))
    return n | 1 if rng.random() < 0.6 else n


def draw(rng):
    op = rng.choice(("sort", "sort", "sort", "pairs", "argsort", "range", "segmented", "plan", "kway", "host"))
    dtype = rng.choice(tuple(WIDTH))
    wide = WIDTH[dtype] == 8
    case = {"op": op, "dtype": dtype, "dist": rng.choice(DISTS)}
    if op == "sort":
        case["n"] = _log_size(rng, 6, 27.5 if wide else 29)
    elif op in ("pairs", "argsort"):
        case["n"] = _log_size(rng, 8, 25 if wide else 26)
        case["value_bytes"] = rng.choice((4, 8))
    elif op == "range":
        case["n"] = _log_size(rng, 8, 25 if wide else 26)
        bits = 8 * WIDTH[dtype]
        case["begin"] = rng.choice((0, 0, rng.randrange(bits // 2)))
        case["end"] = rng.choice((bits, bits, case["begin"] + rng.randrange(8, bits // 2 + 1)))
        case["descending"] = rng.random() < 0.7
        case["value_bytes"] = rng.choice((0, 4, 8))
    elif op in ("segmented", "plan"):
        case["n"] = _log_size(rng, 14, (26 if wide else 27) if op == "segmented" else 20)
        case["segments"] = int(2.0 ** rng.uniform(2, min(17, math.log2(case["n"]) - 3)))
        case["lengths"] = rng.choice(("zipf", "even"))
    elif op == "kway":
        case["n"] = _log_size(rng, 14, 27 if wide else 28)
        case["runs"] = rng.choice((2, 2, 3, 4, 8, 13, 16, 32, 64))
    else:
        case["n"] = _log_size(rng, 10, 24 if wide else 25)
    return case


def _store(dtype):
    return torch.int32 if WIDTH[dtype] == 4 else torch.int64


def _keys(dtype, dist, n, gen):
    """n keys of the distribution, as raw bits (int32 / int64), on the GPU."""
    store, bits = _store(dtype), 8 * WIDTH[dtype]
    dev = "cuda"
    if dtype in ("f32", "f64"):
        real = torch.float32 if dtype == "f32" else torch.float64
        if dist == "uniform":
            x = torch.rand(n, dtype=real, device=dev, generator=gen)
        elif dist == "zipf":  # heavy-tailed positive values, the small ones many times
            x = torch.rand(n, dtype=real, device=dev, generator=gen).clamp_(min=1e-6).pow_(-5.0).floor_()
        elif dist == "few":
            x = torch.randint(0, 1_000_000, (n,), device=dev, generator=gen, dtype=torch.int32).to(real).mul_(0.01)
        else:
            x = torch.randn(n, dtype=real, device=dev, generator=gen)
        if dist == "nearly":
            x = torch.sort(x)[0]
            _swap_some(x, gen)
        # What float columns hold besides: a few zeros of both signs and a few missing values.
        for value in (0.0, -0.0, float("nan")):
            where = torch.randint(0, n, (n // 1000,), device=dev, generator=gen)
            x[where] = value
        return x.view(store)
    low, high = -(1 << (bits - 1)), (1 << (bits - 1)) - 1
    if dist == "uniform":
        return torch.randint(low, high, (n,), device=dev, generator=gen, dtype=store)
    if dist == "few":  # ids below a million: every id many times in a large input
        return torch.randint(0, 1_000_000, (n,), device=dev, generator=gen, dtype=store)
    if dist == "zipf":
        u = torch.rand(n, dtype=torch.float32, device=dev, generator=gen).clamp_(min=1e-6)
        return u.pow_(-5.0).clamp_(max=2.0e9).to(store)
    if dist == "normal":
        real = torch.float32 if bits == 32 else torch.float64
        x = torch.randn(n, dtype=real, device=dev, generator=gen).mul_(2.0 ** (bits - 5))
        return x.to(store) if dtype[0] == "i" else x.to(store) ^ low  # unsigned: centred on the middle of the range
    x = torch.sort(torch.randint(0, high, (n,), device=dev, generator=gen, dtype=store))[0]
    _swap_some(x, gen)
    return x


def _swap_some(x, gen):
    """Exchanges 1 % of the keys with keys elsewhere."""
    a = torch.arange(0, x.numel(), 100, device=x.device)  # one place in every hundred, each taken once
    x[a] = x[a[torch.randperm(a.numel(), device=x.device, generator=gen)]]


def _cut(rng, n, parts, how):
    """Offsets that cut n keys into `parts` pieces (int64, parts + 1)."""
    if how == "zipf":
        lens = np.minimum(rng.zipf(1.2, parts), 1 << 22).astype(np.float64)
        lens = np.floor(lens * (n / lens.sum())).astype(np.int64)
    elif how == "even":
        lens = rng.uniform(0.75, 1.25, parts)
        lens = np.floor(lens * (n / lens.sum())).astype(np.int64)
    else:
        lens = np.floor(rng.dirichlet(np.ones(parts)) * n).astype(np.int64)
    lens[rng.integers(parts)] += n - int(lens.sum())  # what rounding left over
    offs = np.zeros(parts + 1, dtype=np.int64)
    offs[1:] = np.cumsum(lens)
    return offs


def _sorted_runs(dtype, bits, offs):
    """Each run's keys ascending in the engine's order (integers by value; floats hold no NaN here)."""
    out = torch.empty_like(bits)
    for a, b in zip(offs[:-1], offs[1:]):
        run = bits[a:b]
        if dtype == "f32":
            run = torch.sort(run.view(torch.float32))[0].view(torch.int32)
        elif dtype == "f64":
            run = torch.sort(run.view(torch.float64))[0].view(torch.int64)
        elif dtype[0] == "u":
            top = -(1 << (8 * WIDTH[dtype] - 1))
            run = torch.sort(run ^ top)[0] ^ top
        else:
            run = torch.sort(run)[0]
        out[a:b] = run
    return out


def prepare(case, seed):
    mgs = _mgs()
    ctx, stream = _engine()
    op, dtype, n = case["op"], case["dtype"], case["n"]
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    keys = _keys(dtype, case["dist"], n, gen)
    s = {"op": op, "dtype": dtype, "n": n, "ctx": ctx, "stream": stream, "keys": keys}
    temp_bytes = 0
    if op == "host":
        s["array"] = mgs.host_empty(n, dtype)
        host = keys.cpu().numpy().view(s["array"].dtype)
        np.copyto(s["array"], host)
        del s["keys"]
    elif op == "kway":
        if dtype[0] == "f":  # sorted runs of plain numbers: a NaN or a zero's sign has no place in torch's order
            real = keys.view(torch.float32 if dtype == "f32" else torch.float64)
            real.nan_to_num_(nan=1.0)
            real.add_(0.0)  # -0.0 becomes +0.0
        offs = _cut(np.random.default_rng(seed), n, case["runs"], "dirichlet")
        s["keys"] = _sorted_runs(dtype, keys, offs)
        w = WIDTH[dtype]
        s["runs"] = [s["keys"].data_ptr() + w * int(a) for a in offs[:-1]]
        s["lens"] = [int(b - a) for a, b in zip(offs[:-1], offs[1:])]
        temp_bytes = ctx.merge_temp_bytes(dtype, case["runs"], n)
    elif op in ("segmented", "plan"):
        offs = _cut(np.random.default_rng(seed), n, case["segments"], case["lengths"])
        s["offsets"] = torch.from_numpy(offs).cuda()
        s["segments"] = case["segments"]
        temp_bytes = ctx.segmented_sort_temp_bytes(dtype, n, case["segments"])
    elif op in ("pairs", "argsort") or case.get("value_bytes"):
        s["value_bytes"] = case["value_bytes"]
        vtype = torch.int32 if case["value_bytes"] == 4 else torch.int64
        s["values"] = torch.arange(n, device="cuda", dtype=vtype)
        s["work_values"] = torch.empty_like(s["values"])
        temp_bytes = ctx.sort_pairs_temp_bytes(dtype, case["value_bytes"], n)
    else:
        temp_bytes = ctx.sort_temp_bytes(dtype, n)
    if op == "range":
        s.update(begin=case["begin"], end=case["end"], descending=case["descending"],
                 value_bytes=case["value_bytes"])
    if op != "host":
        s["work"] = torch.empty_like(s["keys"])
        s["temp"] = torch.empty(temp_bytes, dtype=torch.uint8, device="cuda")
        s["temp_bytes"] = temp_bytes
    if op == "plan":
        s["plan"] = ctx.plan_segmented(s["work"].data_ptr(), n, s["offsets"].data_ptr(), s["segments"], dtype,
                                       s["temp"].data_ptr(), temp_bytes)
    torch.cuda.synchronize()
    return s


def run(s):
    op, ctx, n, dtype = s["op"], s["ctx"], s["n"], s["dtype"]
    if op == "host":
        # In place on the caller's pinned buffer; a later pass finds it sorted, the copies are the same.
        ctx.sort_host(s["array"])
        return s["array"].view(np.int32 if s["array"].itemsize == 4 else np.int64)
    work, stream = s["work"], s["stream"]
    h = stream.cuda_stream
    temp, temp_bytes = s["temp"].data_ptr(), s["temp_bytes"]
    with torch.cuda.stream(stream):
        if op == "kway":
            ctx.kway_merge_device(s["runs"], s["lens"], work.data_ptr(), dtype, temp, temp_bytes, h)
            return work
        work.copy_(s["keys"])
        if op == "sort":
            ctx.sort_device(work.data_ptr(), n, dtype, temp, temp_bytes, h)
            return work
        if op == "segmented":
            ctx.segmented_sort_device(work.data_ptr(), n, s["offsets"].data_ptr(), s["segments"], dtype, temp,
                                      temp_bytes, h)
            return work
        if op == "plan":
            s["plan"].launch(h)
            return work
        if op == "argsort":
            ctx.argsort_device(work.data_ptr(), s["work_values"].data_ptr(), s["value_bytes"], n, dtype, temp,
                               temp_bytes, h)
            return work, s["work_values"]
        values, value_bytes = s.get("work_values"), s["value_bytes"]
        if values is not None:
            values.copy_(s["values"])
        d_values = values.data_ptr() if values is not None else 0
        if op == "pairs":
            ctx.sort_pairs_device(work.data_ptr(), d_values, value_bytes, n, dtype, temp, temp_bytes, h)
        else:
            ctx.sort_range_device(work.data_ptr(), n, dtype, s["begin"], s["end"], s["descending"], d_values,
                                  value_bytes, temp, temp_bytes, h)
        return work if values is None else (work, values)


def work(case):
    """Every input key and value read once, every output key and value written once. A sort computes nothing."""
    w, n = WIDTH[case["dtype"]], case["n"]
    v = case.get("value_bytes", 0)
    moved = n * (2 * w + (v if case["op"] == "argsort" else 2 * v))
    return {"bytes": moved + 8 * case.get("segments", 0), "flops": 0}
