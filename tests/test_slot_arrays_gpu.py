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
