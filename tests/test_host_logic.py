"""Host-side logic that needs no GPU: the random-draw bookkeeping that keeps later tensors' hash parameters in step with
the reference when an intermediate tensor is skipped, and the shape arithmetic helpers."""
import numpy as np

from doksparse_b200 import util
from oracle import port


def _state():
    s = np.random.get_state()
    return s[1].copy(), s[2]


def test_skipped_map_consumes_the_reference_draws():
    for key_size, n_buckets, n_new in ((1, 1024, 700), (3, 64, 40), (2, 1 << 20, 1)):
        np.random.seed(3)
        port.draw_hash_parameters(n_buckets, key_size)
        want = _state()
        np.random.seed(3)
        util.consume_fresh_map_draws(n_buckets, key_size, n_new)
        got = _state()
        assert (want[0] == got[0]).all() and want[1] == got[1]


def test_skipped_map_that_would_rehash_draws_twice():
    np.random.seed(9)
    port.draw_hash_parameters(1024, 2)
    port.draw_hash_parameters(int(900 * 2.0), 2)          # 900 > int(0.75 * 1024): the reference rebuilds at 1800 buckets
    want = _state()
    np.random.seed(9)
    util.consume_fresh_map_draws(1024, 2, 900)
    got = _state()
    assert (want[0] == got[0]).all() and want[1] == got[1]


def test_nothing_stored_draws_nothing():
    np.random.seed(1)
    before = _state()
    util.consume_fresh_map_draws(1024, 2, 0)
    after = _state()
    assert (before[0] == after[0]).all() and before[1] == after[1]


def test_shape_helpers():
    assert util.next_power_of_2(1) == 1 and util.next_power_of_2(10_000_000) == 1 << 24 and util.next_power_of_2(1 << 20) == 1 << 20
    assert list(util.shape_to_stride((4, 3, 2))) == [6, 2, 1]
    assert util.next_prime(14) == 17 and util.next_prime(17) in (17, 19)


def test_sliced_exchange_geometry():
    """Arena layout of the sliced exchange: slices hold the mean plus eight standard deviations of the binomial row
    count plus a constant, never more than the capacity, start on 256-row boundaries, and the regions of a generation
    do not overlap."""
    import math
    import torch
    from doksparse_b200.sharded import CudaShardOps
    key_row, value_row = ((1,), torch.int64), ((2,), torch.float32)
    for world, cap in ((2, 30000), (8, 1 << 25), (4, 100), (16, 1 << 20), (8, 1)):
        g = CudaShardOps.sliced_geometry(world, cap, key_row, value_row)
        rows = g["slice_rows"]
        mean = cap / world
        assert rows % 256 == 0 and rows >= min(cap, math.ceil(mean + 8 * math.sqrt(mean))) and rows <= (cap + 255) // 256 * 256
        assert rows <= max(256, mean + 8 * math.sqrt(mean) + 64 + 256)
        if cap >= 1 << 25:
            assert rows <= 1.005 * mean                         # the slack is a fraction of a percent for large batches
        sizes, offs = g["sizes"], g["offs"]
        assert sizes[0] >= world * rows * 8 and sizes[1] >= world * rows * 8 and sizes[2] >= world * 8
        assert sizes[3] >= world * rows * 8 and sizes[4] >= world * rows
        assert all(o % 256 == 0 for o in offs) and all(offs[i] + sizes[i] == offs[i + 1] for i in range(4))
        assert g["gen_bytes"] == offs[4] + sizes[4]


def test_a_table_that_is_collected_while_a_ring_is_taken():
    """The cyclic collector can free a table, which gives its ring back, while another table's ring is being made."""
    import threading
    from types import SimpleNamespace
    from unittest import mock
    from doksparse_b200 import cuda_closed_hashmap as M

    rings, made, taken = M._PinnedRings(), [], []

    class Ring:
        def __init__(self, words, device):
            made.append(self)
            if len(made) == 70:                              # in the middle of the second chunk
                rings.give(taken.pop(), device)

        def wait(self, place):
            pass

    with mock.patch.object(M.L, "native", lambda: SimpleNamespace(Ring=Ring)), \
            mock.patch.object(M.torch, "zeros", lambda *shape, **options: range(shape[0])):
        worker = threading.Thread(target=lambda: [taken.append(rings.take(0)) for _ in range(65)], daemon=True)
        worker.start()
        worker.join(timeout=20)
    assert not worker.is_alive()
    assert len(made) == 128 and len(taken) == 64 and len(rings._free[0]) == 64
    assert len(set(map(id, taken + rings._free[0]))) == 128


def test_pieces_of_a_host_batch_hide_their_host_time():
    """A piece costs about 75 us on the host.  Two of them have to move what the link takes that long for, 55 bytes in a
    nanosecond (a lone operation has nothing else to overlap with: less will do)."""
    from types import SimpleNamespace
    import torch
    from doksparse_b200.host_batch import HostBatch

    class Offline(HostBatch):
        def __init__(self):
            self.chunk_rows, self._takes_outputs, self._staged_set_rows = 1 << 22, True, 0
            self.table = SimpleNamespace(_slots=0, remove_rows=None, remove=None, _element_bound=lambda: 0, _rehash_threshold=0.75, n_buckets=1 << 30)

        def _ring(self, *shape):
            pass

        def _execute(self, chunks):
            self.pieces = [[t.shape[0] for _, t in inputs] for inputs, _ in chunks]

    batch = Offline()
    for log2 in range(10, 24):
        for n in (1 << log2, 3 << (log2 - 1)):
            for cols in (1, 2, 4):
                keys, values, flags = torch.empty(n, 1, dtype=torch.long), torch.empty(n, cols), torch.empty(n, dtype=torch.bool)
                ops = {"get": ((keys, values, flags), 9 + 4 * cols), "set": ((keys, values), 8 + 4 * cols), "remove_rows": ((keys, flags), 9)}
                for name, (args, row_bytes) in ops.items():
                    getattr(batch, name)(*args)
                    alone = [p[0] for p in batch.pieces]
                    batch.run([(name, *args)])
                    assert [p[0] for p in batch.pieces] == alone and sum(alone) == n
                    batch.run([(name, *args)] * 2)
                    together = [p[0] for p in batch.pieces]
                    assert sum(together) == 2 * n
                    for pieces, least in ((alone, 3.2e6), (together[:len(together) // 2], 75e-6 * 55e9)):
                        assert len(pieces) <= 4
                        if len(pieces) > 1 and n <= batch.chunk_rows:
                            assert sum(pieces) / len(pieces) * row_bytes >= least
                    if n == 1 << 22:
                        assert len(alone) == 4


def test_a_set_that_raises_leaves_no_staged_rows():
    """Rows staged for a set that never ran would keep later sets from going in pieces."""
    import pytest
    import torch
    from doksparse_b200.host_batch import HostBatch

    class Offline(HostBatch):
        def __init__(self):
            self._staged_set_rows = 0

    batch = Offline()

    def chunks():
        batch._staged_set_rows += 100
        raise ValueError
        yield

    with pytest.raises(ValueError):
        batch._execute(chunks())
    batch._execute([])
    assert batch._staged_set_rows == 0
