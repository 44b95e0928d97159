"""What sets leave behind belongs to the slot array they wrote: maps that share slots, maps that part from one another, sets on
several streams, and the point where the numbers of rows start over."""
import copy

import numpy as np
import pytest
import torch

from oracle import port
from tests.helpers import assert_same_bytes, dev, host
from tests.test_kernel_edges_gpu import params

pytestmark = pytest.mark.gpu

# row numbers in the values' words | stamps in the slots | in an array of their own
VALUES = {"word": (np.float32, 1), "slot": (np.float32, 2), "array": (np.float32, 4)}


def _maps(tombstone_threshold="auto", **kwargs):
    from doksparse_b200 import CudaClosedHashmap
    return CudaClosedHashmap(tombstone_threshold=tombstone_threshold, **kwargs), port.OracleHashmap(**kwargs)


def _both_set(c, o, keys, values):
    c.set(dev(keys), dev(values))
    o.set(keys, values)


def _same(c, o, keys):
    got, found = c.get(dev(keys))
    expected, there = o.get(keys)
    np.testing.assert_array_equal(host(found), there)
    assert_same_bytes(host(got), expected)
    assert c.n_elements == o.n_elements and c.count_live() == o.n_elements


@pytest.mark.parametrize("kind", sorted(VALUES))
@pytest.mark.parametrize("n", [1000, 30000])
def test_a_clone_of_a_map_that_holds_nothing_is_a_map_of_its_own(kind, n):
    dtype, cols = VALUES[kind]
    rng = np.random.default_rng(n)
    values = lambda k: rng.standard_normal((k, cols)).astype(dtype)
    keys = rng.permutation(10 * n)[:n, None]
    a, oa = _maps(n_buckets=1 << 17, key_size=1, **params(1))
    b, ob = a.clone(), port.OracleHashmap(n_buckets=1 << 17, key_size=1, **params(1))
    _both_set(a, oa, keys, values(n))
    _both_set(b, ob, keys[:10] + 10 ** 6, values(10))
    _both_set(a, oa, keys[::-1].copy(), values(n))
    for c, o in ((a, oa), (b, ob)):
        _same(c, o, np.concatenate([keys, keys[:10] + 10 ** 6]))


@pytest.mark.parametrize("kind", sorted(VALUES))
@pytest.mark.parametrize("n", [1000, 30000])
def test_a_rebuilt_map_and_a_clone_that_keeps_the_old_slots(kind, n):
    """Repeated keys in every batch: each of the two has to tell their last rows by the marks in its own slots."""
    dtype, cols = VALUES[kind]
    rng = np.random.default_rng(n)
    values = lambda k: rng.standard_normal((k, cols)).astype(dtype)
    everything = np.arange(n // 2 + 1)[:, None] * 13
    batch = lambda: everything[rng.integers(0, len(everything), n)]
    a, oa = _maps(n_buckets=1 << 17, key_size=1, tombstone_threshold=None, **params(1))
    for _ in range(3):
        _both_set(a, oa, batch(), values(n))
    gone = everything[:: 7].copy()
    np.testing.assert_array_equal(host(a.remove(dev(gone))), oa.remove(gone))
    b, ob = a.clone(), copy.deepcopy(oa)
    tombstones = b.n_tombstones
    a.rebuild()
    assert a.n_tombstones == a.tombstone_bound == 0 and b.n_tombstones == b.tombstone_bound == tombstones > 0
    for _ in range(2):
        for c, o in ((a, oa), (b, ob)):
            _both_set(c, o, batch(), values(n))
            _same(c, o, everything)


@pytest.mark.parametrize("kind", sorted(VALUES))
@pytest.mark.parametrize("n", [700, 20000])
def test_sets_of_different_keys_on_two_streams(kind, n):
    """Each stream sets keys of its own, with repetitions, while the other does; after both, one set of all of them."""
    cols = VALUES[kind][1]
    table, oracle = _maps(n_buckets=1 << 18, key_size=1, **params(1))
    rng = np.random.default_rng(n)
    everything = np.arange(2 * n)[:, None]
    _both_set(table, oracle, everything, np.zeros((2 * n, cols), np.float32))
    streams = [torch.cuda.Stream() for _ in range(2)]
    for _ in range(15):
        rows = (n, n // 9)
        batches = [[(rng.integers(0, n, (rows[s], 1)) + s * n, rng.standard_normal((rows[s], cols)).astype(np.float32)) for _ in range(3)] for s in range(2)]
        on_device = [[(dev(k), dev(v)) for k, v in parts] for parts in batches]
        torch.cuda.synchronize()
        for stream in streams:
            with torch.cuda.stream(stream):
                torch.cuda._sleep(1 << 20)               # until all of the sets are queued
        for k in range(3):
            for s in range(2):
                with torch.cuda.stream(streams[s]):
                    table.set(*on_device[s][k])
        torch.cuda.synchronize()
        for parts in batches:
            for k, v in parts:
                oracle.set(k, v)
        _same(table, oracle, everything)
        _both_set(table, oracle, everything[::-1].copy(), rng.standard_normal((2 * n, cols)).astype(np.float32))
        _same(table, oracle, everything)


@pytest.mark.parametrize("n", [700, 20000])
def test_row_numbers_start_over_while_another_stream_sets(n):
    table, oracle = _maps(n_buckets=1 << 18, key_size=1, **params(1))
    rng = np.random.default_rng(n)
    everything = np.arange(2 * n)[:, None]
    _both_set(table, oracle, everything, np.zeros((2 * n, 1), np.float32))
    streams = [torch.cuda.Stream() for _ in range(2)]
    for _ in range(4):
        batches = [(rng.integers(0, n, (n, 1)) + s * n, rng.standard_normal((n, 1)).astype(np.float32)) for s in (0, 1, 0, 1)]
        on_device = [(dev(k), dev(v)) for k, v in batches]
        torch.cuda.synchronize()
        table._marks.numbered = 0x7ffffff0 - 2 * n + 1           # room for one of the four
        for i in range(4):
            with torch.cuda.stream(streams[i % 2]):
                table.set(*on_device[i])
        assert table._marks.numbered == 3 * n
        torch.cuda.synchronize()
        for k, v in batches:
            oracle.set(k, v)
        _same(table, oracle, everything)


@pytest.mark.parametrize("n", [700, 20000])
@pytest.mark.parametrize("dtype", [np.float32, np.uint8])
def test_replayed_sets_among_others(n, dtype):
    """A set in a graph wins over what came before its replay and loses against what comes after it, whatever numbers the
    slots hold, and reuses tombstones."""
    table, oracle = _maps(n_buckets=1 << 19, key_size=1, **params(1))
    rng = np.random.default_rng(n)
    everything = np.arange(2 * n)[:, None]
    batch = lambda m: (rng.integers(0, 2 * n, (m, 1)), rng.integers(0, 100, (m, 1)).astype(dtype))
    _both_set(table, oracle, *batch(n))
    keys, values = (dev(x) for x in batch(n))
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        table.set(keys, values)
    for i in range(6):
        k, v = batch(n)
        keys.copy_(dev(k))
        values.copy_(dev(v))
        graph.replay()
        oracle.set(k, v)
        _same(table, oracle, everything)
        if i % 2:
            _both_set(table, oracle, *batch(n // 3))
        if i == 2:
            table._marks.numbered = 0x7ffffff0                 # none left, and a replay may be on its way at any time: stamps
        gone = np.unique(rng.integers(0, 2 * n, n // 5))[:, None]
        np.testing.assert_array_equal(host(table.remove(dev(gone))), oracle.remove(gone))
        _same(table, oracle, everything)
    assert table._marks.numbered == 0x7ffffff0 and table._marks.epoch == 2


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
def test_assignment_by_selectors_of_the_general_way(dtype):
    """Lists, arrays, other integer types and values of another type or device, up to eight dims."""
    from doksparse_b200 import SparseDOKTensor
    shape = (3, 2, 4, 2, 3, 2, 2, 5)
    np.random.seed(1)
    t, dense = SparseDOKTensor(shape, dtype=dtype), torch.zeros(shape, device="cuda", dtype=dtype)
    rng = np.random.default_rng(0)
    for _ in range(3):
        i, j = rng.integers(0, 3, 6), torch.from_numpy(rng.integers(0, 5, 6)).to(torch.int32)
        picked = (i.tolist(), 1, slice(1, 3), 0, rng.integers(0, 3, 6), slice(None), 1, j)
        at = tuple(torch.as_tensor(p).cuda().long() if isinstance(p, (list, np.ndarray, torch.Tensor)) else p for p in picked)
        values = torch.randint(0, 100, tuple(t[at].shape))
        t[picked] = values
        for e in range(6):                                       # the last one of equal positions stays
            one = tuple(p[e] if isinstance(p, torch.Tensor) else p for p in at)
            dense[one] = values[e].to("cuda", dtype)
        assert torch.equal(t.to_dense(), dense)


@pytest.mark.parametrize("kind", sorted(VALUES))
@pytest.mark.parametrize("n", [700, 8193, 70000])
@pytest.mark.parametrize("distinct", [1, 3, 300])
def test_rows_that_lost_to_a_later_one_are_counted(kind, n, distinct):
    from doksparse_b200._lib import CNT_DUPLICATES
    table, _ = _maps(n_buckets=1 << 18, key_size=1, **params(1))
    rng = np.random.default_rng(n)
    cols = VALUES[kind][1]
    for _ in range(3):                                           # new keys, then stored ones
        keys = rng.integers(0, distinct, (n, 1)) * 7919
        before = int(table._state[CNT_DUPLICATES])
        table.set(dev(keys), torch.zeros(n, cols, device="cuda"))
        assert int(table._state[CNT_DUPLICATES]) - before == n - len(np.unique(keys))
