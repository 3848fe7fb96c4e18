"""GPU parity of the plain device sort's partition path (partition_sort.cu) where it can go wrong: the sizes at
which it changes from one block to one level and to two levels of cells, and keys that its sampled maps and its
bins fit badly (few values, values crowded over many scales, clusters, one value with a few others, zeros of both
signs). Sorting moves keys and computes none, so outputs are compared with the oracle byte for byte."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

BLOCK = {4: 512 * 20, 8: 512 * 14}  # keys one block of 512 threads sorts; 1024 threads sort twice as many
ONE_LEVEL = {4: 1022 * 3584, 8: 1022 * 2506}  # keys that one level of cells takes at most


def keys(dtype, kind, n, rng):
    dt = np.dtype(dtype)
    if n == 0:
        return np.empty(0, dt)
    bits = 8 * dt.itemsize
    u = np.dtype(f"u{dt.itemsize}")
    full = rng.integers(0, 1 << bits, n, dtype=u, endpoint=False) if bits < 64 else \
        rng.integers(0, (1 << 64) - 1, n, dtype=u, endpoint=True)
    if kind == "uniform":
        out = full
    elif kind == "scales":  # as many keys between 2^k and 2^(k+1) for every k
        out = full >> rng.integers(0, bits, n).astype(u)
    elif kind == "few":
        out = (rng.integers(0, 17, n) * 1000003).astype(u)
    elif kind == "dense":  # every value many times
        out = rng.integers(0, max(2, n // 50), n).astype(u)
    elif kind == "clusters":
        centres = full[:8] if n >= 8 else full
        out = centres[rng.integers(0, len(centres), n)] + rng.integers(0, 300, n).astype(u)
    elif kind == "mostly_one":
        out = np.full(n, 777, dtype=u)
        out[rng.integers(0, n, max(1, n // 500))] = full[:max(1, n // 500)]
    else:  # zeros of both signs, infinities and NaNs among normal values (bit patterns, for every type)
        real = rng.standard_normal(n).astype(np.float32 if bits == 32 else np.float64)
        pick = rng.random(n)
        real[pick < 0.3] = 0.0
        real[pick < 0.15] = -0.0
        real[pick > 0.98] = np.inf
        real[pick > 0.985] = -np.inf
        real[pick > 0.99] = np.nan
        out = real.view(u)
    return out.view(dt)


@pytest.mark.parametrize("dtype", ["u4", "i4", "f4", "u8", "i8", "f8"])
@pytest.mark.parametrize("kind", ["uniform", "scales", "few", "dense", "clusters", "mostly_one", "zeros"])
def test_partition_sort_matches_oracle(ctx, orc, dtype, kind):
    w = np.dtype(dtype).itemsize
    names = {"u4": "u32", "i4": "i32", "f4": "f32", "u8": "u64", "i8": "i64", "f8": "f64"}
    sizes = [2, BLOCK[w], BLOCK[w] + 1, 2 * BLOCK[w], 2 * BLOCK[w] + 1, 150_001, ONE_LEVEL[w], ONE_LEVEL[w] + 1]
    for n in sizes:
        a = keys(dtype, kind, n, np.random.default_rng(n))
        t = torch.from_numpy(a.view(np.int32 if w == 4 else np.int64).copy()).cuda()
        torch.cuda.synchronize()
        ctx.sort_device(t.data_ptr(), n, names[dtype])
        ctx.synchronize()
        assert t.cpu().numpy().view(dtype).tobytes() == orc.sort(a).tobytes(), f"{dtype} {kind} n={n}"


@pytest.mark.parametrize("dtype", ["u4", "i4", "u8", "i8"])
def test_large_integer_segments_match_oracle(ctx, orc, dtype):
    """Segments above one tile of the segmented sort take the partition path for integer keys: every kind of keys,
    lengths at the path's edges, two levels of cells in one segment, empty and small segments between them."""
    w = np.dtype(dtype).itemsize
    tile = {4: 16384, 8: 8192}[w]
    kinds = ["uniform", "scales", "few", "dense", "clusters", "mostly_one", "zeros"]
    lens, parts = [], []
    for i, kind in enumerate(kinds):
        for n in (tile + 1, 0, 5 * tile + i, 37):
            lens.append(n)
            parts.append(keys(dtype, kind, n, np.random.default_rng(100 * i + n)))
    lens += [ONE_LEVEL[w] + 77, 3 * tile]
    parts += [keys(dtype, "uniform", lens[-2], np.random.default_rng(1)), np.full(lens[-1], 5, dtype=dtype)]
    a = np.concatenate(parts)
    offs = np.zeros(len(lens) + 1, dtype=np.uint64)
    offs[1:] = np.cumsum(lens)
    t = torch.from_numpy(a.view(np.int32 if w == 4 else np.int64).copy()).cuda()
    o = torch.from_numpy(offs.view(np.int64)).cuda()
    torch.cuda.synchronize()
    names = {"u4": "u32", "i4": "i32", "u8": "u64", "i8": "i64"}
    ctx.segmented_sort_device(t.data_ptr(), a.size, o.data_ptr(), len(lens), names[dtype])
    ctx.synchronize()
    assert t.cpu().numpy().view(dtype).tobytes() == orc.segmented_sort(a, offs).tobytes()
