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


def heavy_end(kind, n, rng):
    """8-byte keys half of which are the largest (or, mirrored, the smallest) value that a sample of them shows, with a
    few others beyond it that agree with it in their high word and that a sample most likely misses."""
    if kind == "clipped":  # cosine similarities clipped to 1.0, and a few just above it
        a = rng.uniform(0.94, 1.0, n)
        a[rng.permutation(n)[:n // 2]] = 1.0
        a[rng.permutation(n)[:5]] = 1.0 + 2.0 ** -52
    else:  # ids in the high word; low words of their own for a few keys of the most frequent id
        a = rng.integers(0, 100_000, n, dtype=np.uint64) << np.uint64(32)
        heavy = np.uint64(100_000 << 32)
        a[rng.permutation(n)[:n // 2]] = heavy
        a[rng.permutation(n)[:3]] = heavy + np.array([9, 5, 7], dtype=np.uint64)
    return a


def mirrored(a):
    return -a if a.dtype.kind == "f" else ~a


@pytest.mark.parametrize("n", [1 << 20, 2_000_000, 10_000_000])
@pytest.mark.parametrize("kind,dtype", [("clipped", "f8"), ("ids", "u8"), ("ids", "i8"), ("ids", "f8")])
def test_heavy_end_values_match_oracle(ctx, orc, kind, dtype, n):
    a = heavy_end(kind, n, np.random.default_rng(n))
    for b in (a, mirrored(a)):
        b = b.view(dtype)
        assert sorted_on_device(ctx, b).tobytes() == orc.sort(b).tobytes()


@pytest.mark.parametrize("dtype", ["u8", "i8"])
def test_heavy_end_values_in_large_segments_match_oracle(ctx, orc, dtype):
    rng = np.random.default_rng(5)
    parts = []
    for n in (20_000, 1 << 20, 300_001, 3_000_000):
        a = heavy_end("ids", n, rng)
        parts += [a.view(dtype), mirrored(a).view(dtype)]
    a = np.concatenate(parts)
    offs = np.concatenate([[0], np.cumsum([p.size for p in parts])]).astype(np.uint64)
    t = torch.from_numpy(a.view(np.int64).copy()).cuda()
    o = torch.from_numpy(offs.view(np.int64)).cuda()
    torch.cuda.synchronize()
    ctx.segmented_sort_device(t.data_ptr(), a.size, o.data_ptr(), len(parts), NAMES[dtype])
    ctx.synchronize()
    assert t.cpu().numpy().view(dtype).tobytes() == orc.segmented_sort(a, offs).tobytes()


LARGEST = (1 << 32) - 1  # the most keys a sort takes
STEP = 1 << 28


def sort_largest(ctx, fill, dtype):
    """LARGEST 4-byte keys, made and sorted in place on the device; fill(i) gives the keys at positions i."""
    temp_bytes = ctx.sort_temp_bytes(dtype, LARGEST)
    if torch.cuda.mem_get_info()[0] < 4 * LARGEST + temp_bytes + (16 << 30):
        pytest.skip("not enough device memory")
    t = torch.empty(LARGEST, dtype=torch.int32, device="cuda")
    temp = torch.empty(temp_bytes, dtype=torch.uint8, device="cuda")
    for i in range(0, LARGEST, STEP):
        j = min(LARGEST, i + STEP)
        t[i:j] = fill(torch.arange(i, j, device="cuda"))
    torch.cuda.synchronize()
    ctx.sort_device(t.data_ptr(), LARGEST, dtype, temp.data_ptr(), temp_bytes)
    ctx.synchronize()
    return t


def check_largest(t, expected):
    for i in range(0, LARGEST, STEP):
        j = min(LARGEST, i + STEP)
        assert torch.equal(t[i:j], expected(torch.arange(i, j, device="cuda"))), f"[{i}, {j})"


def test_largest_sort_of_distinct_keys(ctx):
    """Every uint32 but one, shuffled by an odd multiplier: the counts of tiles and chunks take nearly all 32 bits."""
    missing = LARGEST * 2654435761 % (1 << 32)
    t = sort_largest(ctx, lambda i: (i * 2654435761).to(torch.int32), "u32")
    check_largest(t, lambda i: (i + (i >= missing)).to(torch.int32))


def test_largest_sort_of_one_value_and_a_few_others(ctx):
    """One value all but 4096 times: its cell is copied in chunks."""
    t = sort_largest(ctx, lambda i: torch.where(i % (1 << 20) == 5, i >> 20, 5000).to(torch.int32), "u32")
    check_largest(t, lambda i: torch.where(i < 4096, i, 5000).to(torch.int32))


def test_largest_sort_of_zeros_of_both_signs(ctx):
    """Zeros of both signs all but 15 times: their signs are written back in input order, over nearly all positions."""
    sign, one = -(1 << 31), 0x3F800000
    zero = lambda i: torch.where(i % 3 == 0, sign, 0)
    t = sort_largest(ctx, lambda i: torch.where(i % STEP == STEP - 1, one, zero(i)).to(torch.int32), "f32")
    others = LARGEST // STEP  # the input position of the i-th zero is i plus the others before it
    check_largest(t, lambda i: torch.where(i >= LARGEST - others, one, zero(i + i // (STEP - 1))).to(torch.int32))


@pytest.mark.parametrize("dtype", ["u4", "i8"])
def test_overlapping_large_segments_are_left_out(ctx, mgs, orc, dtype):
    """Offsets that go back make segments overlap. A large one that starts before an earlier one's end stays as it is
    and is reported; the disjoint ones are sorted, and nothing is written behind the scratch."""
    n = 1 << 20
    rng = np.random.default_rng(6)
    a = rng.integers(0, 1 << 31, n).astype(dtype)
    q = n // 4
    cases = [([0, 2 * q, q, 3 * q, n], [(0, 2 * q), (3 * q, n)]),
             ([0, 3 * q, 0, 3 * q], [(0, 3 * q)]),
             ([0, 3 * q] * 1500 + [3 * q, n], [(0, 3 * q), (3 * q, n)]),
             ([q, 2 * q] + [0, q] * 3 + [2 * q, n], [(q, 2 * q), (2 * q, n)])]
    for offs, kept in cases:
        nseg = len(offs) - 1
        temp_bytes = ctx.segmented_sort_temp_bytes(NAMES[dtype], n, nseg)
        temp = torch.full((temp_bytes + (1 << 20),), 0x5A, dtype=torch.uint8, device="cuda")
        t = torch.from_numpy(a.view(np.int32 if a.itemsize == 4 else np.int64).copy()).cuda()
        o = torch.tensor(offs, dtype=torch.int64, device="cuda")
        torch.cuda.synchronize()
        ctx.segmented_sort_device(t.data_ptr(), n, o.data_ptr(), nseg, NAMES[dtype], temp.data_ptr(), temp_bytes)
        with pytest.raises(mgs.MgsError) as e:
            ctx.synchronize()
        assert e.value.code == mgs.MGS_ERR_INVALID
        want = a.copy()
        for b, c in kept:
            want[b:c] = orc.sort(a[b:c])
        assert t.cpu().numpy().view(dtype).tobytes() == want.tobytes(), offs[:5]
        assert bool((temp[temp_bytes:] == 0x5A).all())


@pytest.mark.parametrize("dtype", ["u8", "i8", "f8"])
def test_ordered_clustered_keys_match_oracle(ctx, orc, dtype):
    """Sorted, reversed and nearly sorted keys whose cells are quantiles of the sample (clusters, heavy tails)."""
    n = 1_500_000
    rng = np.random.default_rng(7)
    clusters = np.sort(rng.integers(0, 1 << 62, 2000))[rng.integers(0, 2000, n)] + rng.integers(0, 3000, n)
    tail = (np.maximum(rng.random(n), 1e-6) ** -2.5).astype(np.int64) << 8
    for a in (np.sort(clusters), np.sort(tail)):
        nearly = a.copy()
        i = rng.permutation(n)[:n // 50]
        nearly[i] = nearly[rng.permutation(i)]
        for b in (a, a[::-1], nearly):
            b = np.ascontiguousarray(b).view(dtype)
            assert sorted_on_device(ctx, b).tobytes() == orc.sort(b).tobytes()


def several_scales(dtype, n, rng):
    """Keys in clusters within clusters: bins and parts of bins hold many different keys, and merges order them."""
    bits = 8 * np.dtype(dtype).itemsize
    top = rng.integers(0, 1 << (bits - 1), 5, dtype=np.uint64)[rng.integers(0, 5, n)]
    mid = rng.integers(0, 1 << (bits // 2), 9, dtype=np.uint64)[rng.integers(0, 9, n)]
    return (top + mid + rng.integers(0, 200, n).astype(np.uint64)).astype(f"u{bits // 8}").view(dtype)


@pytest.mark.parametrize("dtype", ["u4", "i4", "f4", "u8", "i8", "f8"])
def test_keys_clustered_at_several_scales_match_oracle(ctx, orc, dtype):
    """The sizes of one block, its edges and remainders, one and two levels of cells."""
    block = {4: 512 * 20, 8: 512 * 14}[np.dtype(dtype).itemsize]
    item = block // 512
    rng = np.random.default_rng(8)
    for n in (2, item - 1, item + 1, 2 * item, 33 * item + 5, block - 1, block, block + 1, 2 * block - item, 2 * block,
              2 * block + 1, 100_003, 1 << 20, 5_000_011):
        a = several_scales(dtype, n, rng)
        assert sorted_on_device(ctx, a).tobytes() == orc.sort(a).tobytes(), f"{dtype} n={n}"


@pytest.mark.parametrize("dtype,k", [("u4", 3), ("i4", 16), ("u8", 32), ("i8", 64)])
def test_kway_tiles_of_integer_keys_match_oracle(ctx, orc, dtype, k):
    """Merges whose tiles are sorted by bins: dense keys, clusters, one value; one key less and more than whole tiles."""
    w = np.dtype(dtype).itemsize
    tile = {4: 512 * 20, 8: 512 * 14}[w]
    rng = np.random.default_rng(k)
    for total in (k, tile - 1, tile, tile + 1, 5 * tile + 3):
        for a in (several_scales(dtype, total, rng), rng.permutation(total).astype(f"u{w}").view(dtype),
                  np.full(total, 9, dtype=dtype)):
            cuts = np.sort(rng.integers(0, total + 1, k - 1))
            runs = [orc.sort(r) if r.size else r for r in np.split(a, cuts)]
            t = torch.from_numpy(np.concatenate(runs).view(np.int32 if w == 4 else np.int64).copy()).cuda()
            out = torch.empty_like(t)
            starts = np.concatenate([[0], cuts])
            torch.cuda.synchronize()
            ctx.kway_merge_device([t.data_ptr() + w * int(s) for s in starts], [r.size for r in runs], out.data_ptr(),
                                  NAMES[dtype])
            ctx.synchronize()
            assert out.cpu().numpy().view(dtype).tobytes() == orc.sort(a).tobytes(), f"{dtype} k={k} total={total}"


@pytest.mark.parametrize("dtype", ["u8", "i8", "f8"])
def test_grid_barrier_that_runs_out_reports_timeout_and_context_recovers(mgs, orc, dtype):
    """With a bound of one poll, the blocks that reach the last kernel's barrier before the others give up: the sort
    ends with an error status, and the same context sorts again. The heavy value's cell makes the kernel probe its
    keys, which ends at that barrier."""
    a = heavy_end("ids", 1 << 20, np.random.default_rng(3)).view(dtype)
    ctx = mgs.Context(0)
    try:
        t = torch.from_numpy(a.view(np.int64).copy()).cuda()
        torch.cuda.synchronize()
        mgs.inject_waits(0, lookback_spins=1)
        try:
            ctx.sort_device(t.data_ptr(), a.size, NAMES[dtype])
            with pytest.raises(mgs.MgsError) as err:
                ctx.synchronize()
            assert err.value.code == mgs.MGS_ERR_TIMEOUT
            assert "queue" in str(err.value)
        finally:
            mgs.inject_waits(0)
        ctx.synchronize()  # the status was taken
        assert sorted_on_device(ctx, a).tobytes() == orc.sort(a).tobytes()
    finally:
        ctx.close()


def test_autotune_leaves_other_threads_sorts_alone(mgs, orc):
    """The autotuner times onesweep variants; plain sorts that other threads issue meanwhile stay partition sorts."""
    import threading
    a = np.random.default_rng(4).integers(0, 1 << 32, 150_001, dtype=np.uint32)  # a size class that is being tuned
    tuning, mine = mgs.Context(0), mgs.Context(0)
    try:
        mine.set_profiling(True)
        th = threading.Thread(target=tuning.autotune, args=("u32", 3 << 16, 40))
        th.start()
        while th.is_alive():
            assert sorted_on_device(mine, a).tobytes() == orc.sort(a).tobytes()
        th.join()
        names = set(mine.kernel_times())
        assert "part_scatter" in names and "radix_onesweep" not in names
    finally:
        tuning.close()
        mine.close()


@pytest.mark.parametrize("dtype", ["u4", "f4", "u8", "f8"])
def test_scratch_of_the_onesweep_is_enough(ctx, mgs, orc, dtype):
    """The partition sort needs more scratch than the onesweep at many sizes. Scratch that holds only the onesweep's
    state, look-back words and second buffer is still taken, by plain, recorded and range sorts; a byte less is not."""
    name, w = NAMES[dtype], np.dtype(dtype).itemsize
    up = lambda x: (x + 255) // 256 * 256
    rng = np.random.default_rng(9)
    for n in (30_000, 100_000, 1 << 20):
        tile = {4: 4096, 8: 2048}[w]
        least = 16640 + 2 * up((n + tile - 1) // tile * 1024) + up(n * w)
        assert least < ctx.sort_temp_bytes(name, n)
        a = rng.integers(0, 1 << 31, n).astype(f"u{w}").view(dtype)
        temp = torch.full((least + 4096,), 0x5A, dtype=torch.uint8, device="cuda")
        t = torch.empty(n, dtype=torch.int32 if w == 4 else torch.int64, device="cuda")
        keys, want = torch.from_numpy(a.view(np.int32 if w == 4 else np.int64).copy()).cuda(), orc.sort(a).tobytes()

        def check(sort):
            t.copy_(keys)
            torch.cuda.synchronize()
            sort()
            ctx.synchronize()
            assert t.cpu().numpy().tobytes() == want
            assert bool((temp[least:] == 0x5A).all())

        check(lambda: ctx.sort_device(t.data_ptr(), n, name, temp.data_ptr(), least))
        check(lambda: ctx.sort_range_device(t.data_ptr(), n, name, 0, 8 * w, False, 0, 0, temp.data_ptr(), least))
        plan = ctx.plan_sort(t.data_ptr(), n, name, temp.data_ptr(), least)
        try:
            check(plan.launch)
        finally:
            plan.close()
        for refused in (lambda: ctx.sort_device(t.data_ptr(), n, name, temp.data_ptr(), least - 1),
                        lambda: ctx.plan_sort(t.data_ptr(), n, name, temp.data_ptr(), least - 1)):
            with pytest.raises(mgs.MgsError) as err:
                refused()
            assert err.value.code == mgs.MGS_ERR_INVALID
