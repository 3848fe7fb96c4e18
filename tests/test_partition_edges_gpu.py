"""GPU parity of the partition sort (partition_sort.cu) on inputs that sit at the edges of its arithmetic. Sorting
moves keys and computes none, so outputs are compared with the oracle byte for byte."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

NAMES = {"u4": "u32", "i4": "i32", "f4": "f32", "u8": "u64", "i8": "i64", "f8": "f64"}


def sorted_on_device(ctx, a):
    t = torch.from_numpy(a.view(np.int32 if a.dtype.itemsize == 4 else np.int64).copy()).cuda()
    torch.cuda.synchronize()
    ctx.sort_device(t.data_ptr(), a.size, NAMES[a.dtype.str[1:]])
    ctx.synchronize()
    return t.cpu().numpy().view(a.dtype)


@pytest.mark.parametrize("dtype", ["u4", "i4", "f4", "u8", "i8", "f8"])
def test_dense_keys_match_oracle(ctx, orc, dtype):
    """Keys whose range is about their number (row ids, permutations): one bin per value, up to the largest block.
    1024 threads sort up to 20480 4-byte keys with 20480 bins, and up to 14336 8-byte keys with 16384."""
    rng = np.random.default_rng(11)
    u = np.dtype(f"u{np.dtype(dtype).itemsize}")
    for n in (5000, 10240, 10241, 14336, 16384, 16385, 18000, 20000, 20479, 20480):
        for top in {n - 1, 16382, 16383, 16384, 20478, 20479, 20480}:  # the keys' range
            offset = rng.integers(0, 1 << 30)
            ids = np.arange(n) if top == n - 1 else np.append(rng.integers(0, top + 1, n - 2), [0, top])
            a = rng.permutation(ids + offset).astype(u).view(dtype)
            assert sorted_on_device(ctx, a).tobytes() == orc.sort(a).tobytes(), f"{dtype} n={n} range={top}"
