"""Kernels at the sizes where they can go wrong: edges of tiles, remainders, the smallest and the largest of a range."""
import numpy as np
import pytest

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
