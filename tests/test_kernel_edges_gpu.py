"""Kernels at the sizes where they can go wrong: edges of tiles, remainders, the smallest and the largest of a range."""
import numpy as np
import pytest
import torch

from tests.helpers import dev, host
from tests.test_map_gpu import Pair

pytestmark = pytest.mark.gpu


def params(key_size):
    big = [2 ** 59 + 55, 2 ** 58 + 27, 2 ** 57 + 29][:key_size]
    return dict(prime1=[1000003] * key_size, prime2=big, alpha1=[77777, 501, 9001][:key_size], beta1=[5, 7, 9][:key_size],
                alpha2=[2 ** 40 + 15, 2 ** 41 + 21, 2 ** 39 + 7][:key_size], beta2=[11, 13, 17][:key_size])


@pytest.mark.parametrize("n_buckets", [1, 7, 255, 256, 257, 260, 1021, 4096])
@pytest.mark.parametrize("key_size,value_cols", [(1, 2), (3, 4), (2, 31)])     # slots of 32, 64 and more than 128 bytes
def test_chains_of_a_full_table(n_buckets, key_size, value_cols):
    """Up to 64 groups the chain is linear, beyond that it goes by strides first; both have to reach every slot."""
    rng = np.random.default_rng(n_buckets)
    rows = lambda lo, hi: (np.stack([np.arange(lo, hi) * (j + 3) + j for j in range(key_size)], axis=1).astype(np.int64),
                           rng.standard_normal((hi - lo, value_cols)))
    pair = Pair(seed=3, n_buckets=n_buckets, key_size=key_size, rehash_threshold=1.0, **params(key_size))
    pair.set(*rows(0, n_buckets))
    assert pair.c.n_elements == n_buckets and pair.c.n_buckets == n_buckets
    pair.get(rows(0, n_buckets + 50)[0])
    gone = n_buckets // 3
    if gone == 0:
        return
    pair.remove(rows(0, gone)[0])
    pair.get(rows(0, n_buckets + 50)[0])
    pair.set(*rows(n_buckets, n_buckets + gone))
    pair.get(rows(0, n_buckets + gone + 50)[0])


@pytest.mark.parametrize("n_buckets", [1, 7, 255, 257, 260, 1021, 40000])
@pytest.mark.parametrize("key_size", [1, 3, 7])                                # 4, 2 and 1 slots per group
@pytest.mark.parametrize("dtype,cols", [(np.float32, 1), (np.float16, 3), (np.uint8, 7)])
def test_lookups_end_at_groups_that_no_key_went_past(n_buckets, key_size, dtype, cols):
    """Values of at most 7 bytes: every way of placing a key marks the full groups before it, tombstones included."""
    rng = np.random.default_rng(n_buckets + key_size)
    rows = lambda lo, hi: np.stack([np.arange(lo, hi) * (j + 3) + j for j in range(key_size)], axis=1).astype(np.int64)
    values = lambda k: rng.integers(0, 100, (k, cols)).astype(dtype)
    long = lambda v: [v[j % 3] + 2 * (j // 3) for j in range(key_size)]
    pair = Pair(seed=3, n_buckets=n_buckets, key_size=key_size, rehash_threshold=1.0, **{k: long(v) for k, v in params(3).items()})
    most = max(1, 19 * n_buckets // 20)                       # chains of many groups, and empty slots
    half = most // 2
    pair.set(rows(0, half), values(half), assume_unique=True)
    pair.set(rows(half, most), values(most - half))
    everything = rows(0, 2 * n_buckets + 50)
    pair.get(everything)
    gone = most // 3
    if gone:
        pair.remove(rows(0, gone))
        pair.get(everything)
        pair.set(rows(most, most + gone), values(gone))       # into the tombstones
        pair.get(everything)
        pair.c.rebuild()
        pair.get(everything)
    pair.set(rows(most + gone, n_buckets + gone), values(n_buckets - most))
    pair.get(everything)


@pytest.mark.parametrize("n_buckets", [40, 120, 250, 1000])
@pytest.mark.parametrize("key_size", [3, 7])                                   # 2 and 1 slots per group
@pytest.mark.parametrize("unique", [False, True])
def test_keys_of_one_uuid_that_start_in_different_groups(n_buckets, key_size, unique):
    """A column that the uuid does not depend on: a set finds the slot that another key made, and lookups have to as well."""
    from doksparse_b200 import CudaClosedHashmap
    long = lambda v: [v[j % 3] + 2 * (j // 3) for j in range(key_size)]
    drawn = {k: long(v) for k, v in params(3).items()}
    drawn["alpha2"][-1] = 0
    most, joined = 17 * n_buckets // 20, 0
    for first in range(0, 10 * n_buckets, n_buckets):
        table = CudaClosedHashmap(n_buckets=n_buckets, key_size=key_size, rehash_threshold=2.0, tombstone_threshold=None, **drawn)
        keys = (first + torch.arange(most, device="cuda"))[:, None] * torch.arange(3, 3 + key_size, device="cuda")
        table.set(keys, torch.zeros(most, 1, device="cuda"), assume_unique=unique)
        others = keys.clone()
        others[:, -1] += 1
        others = others[:n_buckets // 10]
        values = 1 + torch.arange(len(others), device="cuda", dtype=torch.float32)[:, None]
        table.set(others, values, assume_unique=unique)
        joined += most + len(others) - table.n_elements
        stored, found = table.get(others)
        assert found.all() and torch.equal(stored, values) and table.remove_rows(others).all()
    assert joined > 0


@pytest.mark.parametrize("n", [1, 31, 300, 5000, 70000])
def test_assignment_counts_repeated_new_positions(n):
    """n_elements grows by every selected position that was not stored, repetitions included; the last one's value stays."""
    from doksparse_b200 import SparseDOKTensor
    rng = np.random.default_rng(n)
    np.random.seed(1)
    t = SparseDOKTensor((3000, 3000), dev(rng.integers(0, 3000, (2, 50000))), dev(rng.standard_normal(50000)))
    for _ in range(2):
        i, j = rng.integers(0, 3000, (2, max(1, n // 3)))
        pick = rng.integers(0, len(i), n)
        i, j, v = i[pick], j[pick], rng.standard_normal(n)
        dense = host(t.to_dense())
        stored, before, live, buckets = t.count_items((dev(i), dev(j))), t._nnz(), t.values().numel(), t.storage().n_buckets
        t[dev(i), dev(j)] = dev(v)
        dense[i, j] = v
        before = before if t.storage().n_buckets == buckets else live        # a rehash counts again
        assert t._nnz() == before + n - stored
        np.testing.assert_array_equal(host(t.to_dense()), dense)


@pytest.mark.parametrize("n", [3, 1024, 1025, 8192, 8193, 70000])
@pytest.mark.parametrize("dtype", [np.float32, np.float16, np.int8])
def test_sets_whose_values_carry_the_row(n, dtype):
    """Up to 4 bytes in 32-byte slots: the last row of a key stays, within a batch and across the point where the rows'
    numbers start over; tombstones are reused, and rows of a full table counted."""
    rng = np.random.default_rng(n)
    pair = Pair(seed=5, n_buckets=100000, rehash_threshold=1.0, **params(1))
    values = lambda k: rng.integers(-100, 100, (k, 1)).astype(dtype)
    for spread in (30, 40000, 90000):
        keys = (rng.zipf(1.3, (n, 1)) % spread) * 7919
        pair.set(keys, values(n))
        pair.get(np.arange(100000)[:, None] * 7919)
        if spread == 40000:
            pair.remove(keys[: n // 3])
            pair.c._marks.numbered = 0x7ffffff0 - n // 2          # the next set's numbers do not fit any more
    full = np.arange(160000)[:, None] * 13 + 10 ** 12
    pair.c.set_rows(dev(np.concatenate([full, full[:5]])), dev(np.concatenate([values(160000)] + [values(5)])))
    stored = pair.c.get(dev(full))[1].cpu().numpy()
    assert pair.c.last_set_failed == (~stored).sum() + (~stored[:5]).sum() > 0
    assert pair.c.nonempty_mask.all()


@pytest.mark.parametrize("n", [3, 1025, 8192, 8193, 70000])
def test_assignment_of_narrow_values_counts_repeated_new_positions(n):
    from doksparse_b200 import SparseDOKTensor
    rng = np.random.default_rng(n)
    np.random.seed(1)
    t = SparseDOKTensor((900, 700), dev(rng.integers(0, 700, (2, 20000))), dev(rng.standard_normal(20000).astype(np.float32)))
    for distinct in (1, n // 3, n):
        i, j = rng.integers(0, 900, distinct), rng.integers(0, 700, distinct)
        pick = rng.integers(0, distinct, n)
        i, j, v = i[pick], j[pick], rng.standard_normal(n).astype(np.float32)
        dense = host(t.to_dense())
        stored, before, live, buckets = t.count_items((dev(i), dev(j))), t._nnz(), t.values().numel(), t.storage().n_buckets
        t[dev(i), dev(j)] = dev(v)
        dense[i, j] = v
        before = before if t.storage().n_buckets == buckets else live        # a rehash counts again
        assert t._nnz() == before + n - stored
        np.testing.assert_array_equal(host(t.to_dense()), dense)


def test_a_captured_set_counts_on_when_it_is_replayed():
    from doksparse_b200 import CudaClosedHashmap
    n = 20000
    table = CudaClosedHashmap(n_buckets=1 << 18, device="cuda:0")
    keys, values = torch.arange(n, device="cuda")[:, None] % 9000, torch.rand(n, 1, device="cuda")
    table.set(keys, values)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        table.set(keys, values)
    for _ in range(3):
        order = torch.randperm(n, device="cuda")
        keys.copy_(keys[order].clone())
        values.copy_(torch.rand(n, 1, device="cuda"))
        graph.replay()
        last = torch.full((9000,), -1, device="cuda").scatter_reduce(0, keys[:, 0], torch.arange(n, device="cuda"), "amax")
        got, found = table.get(torch.arange(9000, device="cuda")[:, None])
        assert bool(found.all()) and torch.equal(got, values[last])


def _rows(rng, kind, n):
    if kind == "i64":
        return rng.integers(-2 ** 62, 2 ** 62, (n, 1))
    if kind == "i64 close":                       # equal leading bits, runs that need a look at the whole row
        return (rng.integers(-2 ** 30, 2 ** 30, (n, 1)) << 24) + rng.integers(0, 3, (n, 1))
    if kind == "i64 clustered":                   # thousands of different rows with equal leading bits
        return (rng.integers(0, 2, (n, 1)) << 60) + rng.integers(0, 4 * n, (n, 1))
    if kind == "i64x3":
        return rng.integers(-5, 40, (n, 3))
    if kind == "i32x4":
        return rng.integers(-2 ** 31, 2 ** 31, (n, 4)).astype(np.int32)
    if kind == "u8x5":
        return rng.integers(0, 8, (n, 5)).astype(np.uint8)
    if kind == "one":
        return np.full((n, 2), 7, np.int16)
    return np.round(rng.uniform(-3000, 3000, (n, 3))).astype(np.float32)


@pytest.mark.parametrize("kind", ["i64", "i64 close", "i64 clustered", "i64x3", "i32x4", "u8x5", "one", "f32x3"])
@pytest.mark.parametrize("n", [1, 2, 33, 1024, 1025, 4096, 4097, 8193, 70001])
def test_removal_of_sorted_unique_rows(kind, n):
    """One block up to 4096 rows, radix passes over tiles of 4096 and 1024 rows beyond; half of the rows are stored."""
    rng = np.random.default_rng(n)
    stored = _rows(rng, kind, n)
    pair = Pair(seed=n, n_buckets=1 << 18)
    pair.set(stored, rng.standard_normal((n, 1)))
    batch = np.concatenate([stored[rng.integers(0, n, n - n // 2)], _rows(rng, kind, n)[:n // 2]])
    flags = pair.remove(batch)
    assert flags.shape[0] == np.unique(batch, axis=0).shape[0]
    pair.get(stored)


def _rows_alike(rng, kind, n):
    """Rows whose leading 32 bits do not tell them apart."""
    wide = lambda *shape: rng.integers(-2 ** 62, 2 ** 62, shape)
    if kind == "zipf 2^34":                        # a few bits more than 32, the small ids in most rows
        return np.minimum(rng.zipf(1.1, (n, 1)), 2 ** 34 - 1 - rng.integers(0, 9, (n, 1)))
    if kind == "whole f32x3":
        return rng.integers(-500, 500, (n, 3)).astype(np.float32)
    if kind == "whole f64 and halves":
        return (rng.integers(-10 ** 6, 10 ** 6, (n, 2)) / 2).astype(np.float64)
    if kind == "f16x5":
        return rng.integers(-300, 300, (n, 5)).astype(np.float16)
    if kind == "zeros of both signs":
        return (rng.integers(-12, 12, (n, 4)) * rng.choice([-2.0 ** 20, 2.0 ** 20], (n, 4))).astype(np.float32)
    if kind == "few leading values":               # 62 + 62 bits: four words
        return np.concatenate([wide(7, 1)[rng.integers(0, 7, n)], wide(n // 2 + 1, 1)[rng.integers(0, n // 2 + 1, n)]], axis=1)
    if kind == "all words":                        # 8 columns of 64 bits, the last ones different
        return np.concatenate([wide(1, 6)[np.zeros(n, int)] + rng.integers(0, 2, (n, 6)) * 2 ** 61, wide(n, 2)], axis=1)
    if kind == "last word":
        return np.concatenate([wide(2, 2)[rng.integers(0, 2, n)], rng.integers(0, 3 * n, (n, 1))], axis=1)
    rows = wide(n, 1)                              # scattered, and ...
    if kind == "popular":                          # ... runs of one key's repetitions and a few others
        for k in range(40):
            rows[k * (n // 60):(k + 1) * (n // 60)] = rows[-1 - k]
            rows[k * (n // 60):k * (n // 60) + k % 31] += np.arange(1, k % 31 + 1)[:, None]
    if kind == "clumps":                           # ... runs of many different rows
        for k, m in enumerate((16, 17, 200, 900, 1100)):
            rows[k * (n // 6):k * (n // 6) + min(m, n // 6)] = (rows[-1 - k] >> 13 << 13) + rng.integers(0, 4 * m, (min(m, n // 6), 1))
    if kind == "short runs":
        rows[:3000] = (rows[:3000] // 64) * 64 + rng.integers(0, 64, (3000, 1))
        rows[:3000] = np.repeat(rows[:60], 50, axis=0) + rng.integers(0, 40, (3000, 1))
    return rows[rng.permutation(n)]


@pytest.mark.parametrize("kind", ["zipf 2^34", "whole f32x3", "whole f64 and halves", "f16x5", "zeros of both signs", "few leading values", "all words", "last word",
                                  "popular", "clumps", "short runs"])
@pytest.mark.parametrize("n", [4097, 8193, 70001, 700001])
def test_removal_of_rows_with_equal_leading_bits(kind, n, monkeypatch):
    """Sorted by every word of the packed rows, or by the first and its runs put in order; not by the library."""
    rng = np.random.default_rng(n)
    rows = _rows_alike(rng, kind, n)
    half = rows[:n // 2]
    pair = Pair(seed=n, n_buckets=1 << 21)
    pair.set(half, rng.standard_normal((len(half), 1)))
    for library in (torch, torch.Tensor):
        monkeypatch.setattr(library, "unique", None)
    flags = pair.remove(rows)
    assert flags.shape[0] == np.unique(rows, axis=0).shape[0]
    pair.get(rows[:5000])


def test_removal_flags_hold_no_memory_of_repeated_rows():
    from doksparse_b200 import CudaClosedHashmap
    np.random.seed(1)
    t = CudaClosedHashmap(n_buckets=1 << 12)
    keys = torch.arange(1000, device="cuda")[:, None]
    t.set(keys, torch.ones(1000, 1, device="cuda"))
    flags = t.remove(keys.repeat(1100, 1))
    assert flags.shape == (1000,) and flags.all() and flags.untyped_storage().nbytes() == 1000


@pytest.mark.parametrize("n", [100, 6000])
def test_removal_of_rows_with_nans(n):
    from doksparse_b200 import CudaClosedHashmap
    np.random.seed(1)
    t = CudaClosedHashmap(n_buckets=1 << 16)
    keys = torch.arange(2 * n, device="cuda").reshape(n, 2).float()
    t.set(keys, torch.ones(n, 1, device="cuda"))
    keys[n // 2, 1] = float("nan")
    before = t.n_elements
    assert t.remove(keys).shape[0] == n and t.n_elements < before


@pytest.mark.parametrize("dtype", [np.float16, np.float32, np.float64])
def test_distinct_new_rows_of_float_keys(dtype):
    """-0.0 equals 0.0, a stored row is not new, rows that share a uuid count each."""
    pair = Pair(seed=2, n_buckets=1 << 16)
    rng = np.random.default_rng(0)
    first = (rng.integers(-40, 40, (3000, 2)) / 4).astype(dtype)
    pair.set(first, rng.standard_normal((3000, 1)))
    second = np.concatenate([-first[:500], first[500:1500] * 0, (rng.integers(-60, 60, (5000, 2)) / 4).astype(dtype)])
    pair.set(second, rng.standard_normal((len(second), 1)))


_SELECTORS = {"int": (3,), "negative slice": (slice(-3, None), slice(2, -2)), "column": (slice(None), 257), "last": (slice(None), slice(None), 2),
              "all ints": (6, 299, 4), "pairs": (np.arange(7), np.arange(7) * 40), "outer": (np.arange(3)[:, None], slice(5, 9), np.arange(4)[None]),
              "mask": (slice(1, 3), np.arange(300) % 7 == 0), "mask 2-d": (np.arange(2100).reshape(7, 300) % 11 == 0, slice(0, 2)),
              "empty slice": (slice(5, 2),), "beyond": (slice(4, 100), 3), "0-d": (np.int64(2), slice(0, 4)), "bare slice": slice(1, 4)}


@pytest.mark.parametrize("name", sorted(_SELECTORS))
def test_native_selectors_agree_with_the_general_ones(name):
    """Extents that differ in every dim; the same selection through normalise_selectors is the oracle."""
    from doksparse_b200 import SparseDOKTensor
    from doksparse_b200.selectors import normalise_selectors
    shape = (7, 300, 5)
    np.random.seed(1)
    rng = np.random.default_rng(0)
    dense = torch.from_numpy((rng.random(shape) < 0.4) * rng.standard_normal(shape)).cuda()
    selectors = _SELECTORS[name]
    on_device = lambda s: torch.from_numpy(np.asarray(s)).cuda() if isinstance(s, (np.ndarray, np.integer)) else s
    selectors = on_device(selectors) if not isinstance(selectors, tuple) else tuple(on_device(s) for s in selectors)
    t = SparseDOKTensor.from_dense(dense)
    index, scalars = normalise_selectors(selectors, shape, torch.device("cuda:0"))
    expected = dense[tuple(index)]
    squeezed = expected
    for i in reversed(scalars):
        squeezed = squeezed.squeeze(i) if i < squeezed.ndim and squeezed.shape[i] == 1 else squeezed
    got = t[selectors]
    assert got.shape == squeezed.shape and torch.equal(got, squeezed)
    for values in (torch.randn(expected.shape, device="cuda", dtype=torch.float64), 2.5):
        t[selectors] = values
        dense[tuple(index)] = values
        assert torch.equal(t.to_dense(), dense)


@pytest.mark.parametrize("dtype", [torch.float32, torch.float16, torch.uint8, torch.float64])
@pytest.mark.parametrize("shape,density", [((1,), 1.0), ((2047,), 0.5), ((2048, 3), 1.0), ((129, 17, 5), 0.02), ((700, 1500), 0.001), ((1300, 1000), 0.4)])
def test_dense_round_trip(dtype, shape, density):
    """Few, all and many non-zeros, on fewer elements than a wave takes and on more."""
    from doksparse_b200 import SparseDOKTensor
    np.random.seed(2)
    rng = np.random.default_rng(1)
    dense = torch.from_numpy((rng.random(shape) < density) * rng.integers(1, 100, shape)).cuda().to(dtype)
    t = SparseDOKTensor.from_dense(dense)
    assert t._nnz() == int((dense != 0).sum())
    assert torch.equal(t.to_dense(), dense) and torch.equal(t.to_sparse_coo().to_dense(), dense)
    if len(shape) > 1:
        assert torch.equal(t.transpose(0, 1).to_dense(), dense.transpose(0, 1))


@pytest.mark.parametrize("dtype", [torch.uint8, torch.bfloat16, torch.float32, torch.int64])
@pytest.mark.parametrize("numel", [1, 15, 513, 4097, 700001, 1 << 21])
@pytest.mark.parametrize("density", [0.003, 0.1, 0.14])                 # the list holds an eighth, or 65,536
@pytest.mark.parametrize("offset", [0, 1])                              # not on a 16-byte boundary: the other way
def test_dense_tensor_by_the_list_of_its_non_zeros(dtype, numel, density, offset):
    from doksparse_b200 import SparseDOKTensor
    np.random.seed(2)
    g = torch.Generator(device="cuda").manual_seed(numel)
    dense = torch.randint(1, 100, (numel + offset,), generator=g, device="cuda").to(dtype)
    dense *= (torch.rand(numel + offset, generator=g, device="cuda") < density).to(dtype)
    dense = dense[offset:]
    dense[-1] = 7
    if dtype.is_floating_point:
        dense[0] = -0.0 if numel > 1 else 7
    t = SparseDOKTensor.from_dense(dense)
    assert t._nnz() == int((dense != 0).sum()) and torch.equal(t.to_dense(), dense)


@pytest.mark.parametrize("numel", [255, 256, 257, 2049, 148 * 4 * 2048 + 1, 4 * 148 * 4 * 2048 + 300])
@pytest.mark.parametrize("counts", [(31,), (32,), (33,), (31, 1, 0, 33), (256, 0, 1)])
def test_dense_lists_of_a_warp(numel, counts):
    """A warp takes spans of 256 elements and inserts whenever it has found 32 non-zeros; `counts` in its spans, in turn."""
    from doksparse_b200 import SparseDOKTensor
    np.random.seed(2)
    at = torch.arange(numel, device="cuda")
    order = (at * 37) % 256                                  # where the non-zeros of a span lie
    share = torch.tensor(counts, device="cuda")[(at // 256) // (148 * 4 * 8) % len(counts)]
    dense = torch.where(order < share, at + 1, 0)
    t = SparseDOKTensor.from_dense(dense)
    assert t._nnz() == int((dense != 0).sum()) and torch.equal(t.to_dense(), dense)


@pytest.mark.parametrize("n", [1, 31, 33, 257, 148 * 3 * 256 - 1, 148 * 4 * 256 + 33, 400_003])
@pytest.mark.parametrize("key_cols,value_dtype,value_cols", [(1, torch.float32, 4), (4, torch.float32, 1), (3, torch.int64, 4), (1, torch.uint8, 11),
                                                             (8, torch.float16, 3), (2, torch.float64, 12)])
def test_lookups_over_warp_shares(n, key_cols, value_dtype, value_cols):
    """Slots of 32, 64 and 128 bytes, values in and beyond the word behind the tag; one row per lane, and many."""
    from doksparse_b200 import CudaClosedHashmap
    np.random.seed(4)
    stored = 50_000
    table = CudaClosedHashmap(n_buckets=60_000, rehash_threshold=0.9)
    of = lambda c: torch.stack([c * (2 * j + 3) + 10 ** 6 * j for j in range(key_cols)], dim=1).contiguous()
    all_values = torch.randint(0, 200, (stored, value_cols), device="cuda").to(value_dtype)
    table.set(of(torch.arange(stored, device="cuda")), all_values, assume_unique=True)
    query = torch.randint(0, 2 * stored, (n,), device="cuda")
    values, found = table.get(of(query))
    assert torch.equal(found, query < stored)
    assert torch.equal(values[found], all_values[query[found]]) and not values[~found].any()
    values, _ = table.get(of(query), fallback_value=7)
    assert (values[~found] == 7).all() and torch.equal(values[found], all_values[query[found]])


@pytest.mark.parametrize("n", [148 * 256 - 1, 148 * 256, 148 * 256 * 6 - 1, 148 * 256 * 6, 148 * 256 * 8 - 1, 148 * 256 * 8])
@pytest.mark.parametrize("key_cols,value_dtype,value_cols", [(1, torch.float32, 4), (4, torch.float32, 1), (1, torch.int64, 5), (2, torch.float64, 12)])
def test_lookups_where_the_form_changes(n, key_cols, value_dtype, value_cols):
    """One row per thread below two rows for each lane of the resident warps, shares of the batch from there (and, for narrow
    values, below a block per SM)."""
    test_lookups_over_warp_shares(n, key_cols, value_dtype, value_cols)


@pytest.mark.parametrize("n", [1, 2, 1024, 1025, 2049, 8192, 8193, 65535, 65537, 200_001])
@pytest.mark.parametrize("value_cols", [2, 4, 31])              # stamps in the slot, in an array of their own, slots wider than a line
def test_sets_with_repeated_keys(n, value_cols):
    """One cluster up to 8192 rows, two kernels beyond; a filter of the conflicts from 65536 rows on."""
    pair = Pair(seed=n, n_buckets=1 << 19, **params(1))
    rng = np.random.default_rng(n)
    for spread in (3 * n + 1, n // 50 + 1):
        keys = rng.integers(0, spread, (n, 1))
        pair.set(keys, rng.standard_normal((n, value_cols)))
        pair.get(keys)


@pytest.mark.parametrize("value_cols", [4, 10])
@pytest.mark.parametrize("offset", [0, 2])
def test_lookups_into_outputs_that_are_only_8_byte_aligned(value_cols, offset):
    from doksparse_b200 import CudaClosedHashmap
    np.random.seed(5)
    n = 5000
    table = CudaClosedHashmap(n_buckets=1 << 14)
    keys, stored = torch.arange(n, device="cuda")[:, None] * 3, torch.randn(n, value_cols, device="cuda")
    table.set(keys, stored)
    values = torch.empty(n * value_cols + offset, device="cuda")[offset:].reshape(n, value_cols)
    out, found = table.get(keys, values=values)
    assert found.all() and torch.equal(out, stored) and out.data_ptr() == values.data_ptr()


@pytest.mark.parametrize("key_size", [1, 2, 3, 4, 6])
@pytest.mark.parametrize("dtype,cols", [(torch.uint8, 27), (torch.float16, 13), (torch.float32, 3), (torch.float32, 7), (torch.int64, 2), (torch.int64, 5), (torch.int64, 8)])
@pytest.mark.parametrize("n", [399999, 900001, 1000001])                        # on either side of the rule for wide values
@pytest.mark.parametrize("n_buckets", [1 << 17, (1 << 23) + 77])
def test_lookups_of_wide_values(key_size, dtype, cols, n, n_buckets):
    """Hits and misses of values that end in the first, second and third 32 bytes of their slot, tombstones among them."""
    from doksparse_b200 import CudaClosedHashmap
    if n_buckets > 1 << 17 and (key_size not in (1, 2, 6) or n == 399999):
        pytest.skip("the larger table once per width of slots")
    np.random.seed(1)
    table = CudaClosedHashmap(n_buckets=n_buckets, rehash_threshold=0.95, tombstone_threshold=None)
    stored = n_buckets * 4 // 5 if n_buckets == 1 << 17 else 200001
    keys = lambda c: c[:, None] * torch.arange(3, 3 + key_size, device="cuda") + torch.arange(key_size, device="cuda")
    values = torch.randint(0, 100, (stored, cols), device="cuda").to(dtype)
    table.set(keys(torch.arange(stored, device="cuda")), values, assume_unique=True)
    assert table.remove_rows(keys(torch.arange(0, stored, 5, device="cuda"))).all()
    asked = torch.randint(0, 2 * stored, (n,), device="cuda")
    expected = (asked < stored) & (asked % 5 != 0)
    got, found = table.get(keys(asked), torch.full((cols,), 7, device="cuda", dtype=dtype))
    assert torch.equal(found, expected)
    assert torch.equal(got, torch.where(expected[:, None], values[asked.clamp(max=stored - 1)], 7))


def _looked_at(numel, elem_bytes):
    """Positions of the sample that decides whether the non-zeros of a dense tensor are listed."""
    each, piece = 16 // elem_bytes, np.arange(1024, dtype=np.uint64)
    spacing = np.uint64(numel // each // 1024)
    first = piece * spacing + (spacing * (piece * np.uint64(0x9e3779b1) % np.uint64(1 << 32)) >> np.uint64(32))
    return (first[:, None].astype(np.int64) * each + np.arange(each)).ravel()


@pytest.mark.parametrize("dtype", [torch.uint8, torch.float16, torch.float32, torch.float64])
@pytest.mark.parametrize("numel", [70001, (1 << 20) + 3, 1 << 22])
@pytest.mark.parametrize("kind", ["only there", "all but there", "full", "none", "second half"])
def test_dense_tensors_whose_sample_misleads(dtype, numel, kind):
    from doksparse_b200 import SparseDOKTensor
    np.random.seed(2)
    there = torch.zeros(numel, dtype=torch.bool, device="cuda")
    there[dev(_looked_at(numel, dtype.itemsize))] = True
    at = torch.arange(numel, device="cuda")
    nonzero = {"only there": there, "all but there": ~there & (at % 7 == 0), "full": at >= 0, "none": at < 0, "second half": at >= numel // 2}[kind]
    dense = torch.where(nonzero, at % 100 + 1, 0).to(dtype)
    t = SparseDOKTensor.from_dense(dense)
    assert t._nnz() == int(nonzero.sum()) and torch.equal(t.to_dense(), dense)


@pytest.mark.parametrize("density", [0.01, 0.3, 1.0])
def test_memory_of_a_dense_tensors_conversion(density, monkeypatch):
    """No list beside a table that needs the room: above an eighth of non-zeros there is none, and below it is dropped."""
    from doksparse_b200 import CudaClosedHashmap, SparseDOKTensor
    numel = 1 << 24
    dense = (torch.rand(numel + 1, device="cuda") < density).float()
    peaks = []
    for start in (1, 0):                                         # off a 16-byte boundary: without a list
        torch.cuda.reset_peak_memory_stats()
        before = torch.cuda.memory_allocated()
        SparseDOKTensor.from_dense(dense[start:start + numel])
        peaks.append(torch.cuda.max_memory_allocated() - before)
    assert peaks[1] <= peaks[0] + (numel + 4096 if density < 0.125 else 4096)
    allocate, calls = CudaClosedHashmap._allocate, []

    def short_of_memory(self, *args):
        calls.append(torch.cuda.memory_allocated())
        if len(calls) == 1:
            raise torch.OutOfMemoryError("no room beside the list")
        return allocate(self, *args)

    monkeypatch.setattr(CudaClosedHashmap, "_allocate", short_of_memory)
    if density < 0.125:
        t = SparseDOKTensor.from_dense(dense[:numel])
        assert torch.equal(t.to_dense(), dense[:numel]) and calls[0] - calls[1] >= numel
    else:
        with pytest.raises(torch.OutOfMemoryError):
            SparseDOKTensor.from_dense(dense[:numel])
