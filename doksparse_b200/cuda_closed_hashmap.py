"""CudaClosedHashmap: the reference's batched GPU hash map
(sparse_dok/components/cuda_closed_hashmap.py) with the same constructor, methods, attributes and
error behaviour, on top of libdoksparse.so.

What is kept from the reference
  * key identity is the 64-bit uuid; uuids are bit-identical for identical parameters and keys;
  * parameters are drawn lazily from the global numpy random state with the reference's calls and
    in the reference's order (:66-113, :350-357), so a seeded run draws the same parameters;
  * set / get / remove / rehash bookkeeping: n_elements, n_buckets, rehash trigger and new size
    (:363-366), `remove` dedups with `unique(dim=0)` and returns flags for the sorted unique rows
    (:438-454), `set` returns None (:384), RuntimeError("store something first") (:391-392).
What is different (the slot layout is not part of the contract)
  * `_uuid`, `_values` and `_keys` are strided views (reference shapes) of ONE interleaved slot array: tag, value
    and key row of a slot share a 128-byte line, the unit that a random access costs on B200;
  * the start slot comes from a mixer of the uuid and of alpha1/beta1, not from the reference's first hash
    (prime1 is still drawn, to keep the random stream aligned with the reference);
  * duplicates inside one `set` batch resolve deterministically to the last row.
"""
import ctypes
import math
from collections import namedtuple

import numpy as np
import torch
from torch import Tensor

from . import _lib as L
from .util import next_prime

_PARAM_NAMES = ("prime1", "prime2", "alpha1", "alpha2", "beta1", "beta2")

# The counters of a table, one device int64 array (`_state`): kernels add to a block of L.N_COUNTERS each, and what the
# map reports is a sum over them, so no operation needs counters of its own, their zeroing, or kernels that add them up.
_STATE_WORDS = 32
_BY_SET, _BY_REMOVE, _BY_ROWS, _BY_BULK = 0, 8, 16, 24      # set | remove | distinct new rows of float keys | bulk inserts
_ADJUST = 7              # what n_elements differs by from the slots in use (the reference's DOK assignments over-count)
_COUNTED_NEW = 23        # result of the exact count of a set that may have to grow the table


class _PinnedRings:
    """Pinned landing places for copies of the counters, 8 per table, cut from chunks that serve 64 tables: pinning memory
    takes milliseconds (33 ms once the process has mapped a few GB), more than anything else a new table does.  A table
    gives its ring back when it goes; about 256 are kept.

    No lock: `give` runs where the cyclic collector frees a table, which can be in the middle of `take` on the same thread.
    Taking from and adding to the end of a list are single steps; two threads that both find it empty make a chunk each."""

    def __init__(self):
        self._free = {}

    def take(self, device):
        free = self._free.setdefault(device, [])
        try:
            ring = free.pop()
        except IndexError:
            chunk = torch.zeros(64, 8 * _STATE_WORDS, dtype=torch.long, pin_memory=True)
            rings = [L.native().Ring(words, device) for words in chunk]
            ring = rings.pop()
            free.extend(rings)
        ring.wait(-1)                   # the previous owner's copies have landed: nothing writes here any more
        return ring

    def give(self, ring, device):
        free = self._free[device]
        if len(free) < 256:
            free.append(ring)


_rings = _PinnedRings()


class _Shared:
    """What the maps of one slot array (shallow clones, views) must see together besides its counters and marks: the
    host-side upper bound of n_elements that lets `set` skip a device synchronisation."""
    __slots__ = ("bound", "base", "snapshots", "ring", "device", "known")

    def __init__(self, bound=0):
        self.bound, self.base = bound, bound
        self.snapshots, self.ring, self.device = [], None, None
        self.known = False              # the bound is n_elements itself

    def __del__(self):
        if self.ring is not None and _rings is not None:         # (None: the interpreter is going down)
            _rings.give(self.ring, self.device)

    def exact(self, n):
        """n_elements is known to be n, and nothing enqueued later has been counted in."""
        self.snapshots.clear()
        self.bound = self.base = n
        self.known = True


_Layout = namedtuple("_Layout", "slot_bytes slots_per_group value_offset key_offset stamp_offset n_slots total_bytes")


class CudaClosedHashmap:
    def __init__(
        self,
        n_buckets=1024,
        device="cuda:0",
        prime1=None,
        prime2=None,
        alpha1=None,
        alpha2=None,
        beta1=None,
        beta2=None,
        key_size=None,
        key_perm=None,
        rehash_factor=2.0,
        rehash_threshold=0.75,
        tombstone_threshold="auto",
    ):
        self._empty_marker = -1
        self._removed_marker = -3
        self._n_buckets = int(n_buckets)
        self.device = torch.device(device)
        if self.device.type != "cuda":
            raise L.DokError("CudaClosedHashmap needs a CUDA device: there is no CPU path")
        if not torch.cuda.is_initialized():
            torch.cuda.init()
        L.lib()  # fail loudly now if the extension is missing
        # before the first `set` only the tags exist (cuda_closed_hashmap.py:40)
        self._slots = None           # uint8 storage of the slot array
        self._key_shape = None
        self._key_dtype = None
        self._shared = _Shared()
        self._marks = None           # what sets have left in the slot array (_native.Marks)
        self._value_shape = None
        self._value_dtype = None

        self._key_size = key_size
        # hash parameters: host integers (`_host`) and, where the caller asks for them, device tensors (`_on_device`)
        self._host, self._on_device = {}, {}
        for name, given in zip(_PARAM_NAMES, (prime1, prime2, alpha1, alpha2, beta1, beta2)):
            if isinstance(given, Tensor):
                self._on_device[name] = given
            elif given is not None:
                self._host[name] = [int(v) for v in np.asarray(given).reshape(-1).tolist()]
        self._counters_of_table = None
        self._rehash_factor = rehash_factor
        self._rehash_threshold = rehash_threshold
        # Tombstone-aware maintenance (no counterpart in the reference, whose rehash looks at live items only,
        # cuda_closed_hashmap.py:365: under insert / remove churn its empty slots run out, miss lookups walk ever longer
        # chains, and with none left they walk the whole table).  A removal that leaves live + tombstone slots above
        # t * n_buckets rebuilds the table IN PLACE: same size, same hash parameters (nothing is drawn from the random
        # state), same contents, no tombstones -- invisible to the caller except through `n_tombstones` and `_uuid`.
        # "auto" (the default): t = 0.95, and only once the tombstones are worth a rebuild (2 % of the buckets).
        # None: never (the reference's behaviour).  A number: that t, for any number of tombstones.
        self._tombstone_threshold = tombstone_threshold
        self._tombstone_host_bound = 0          # upper bound on the host of what `tombstone_bound` counts on the device

        self._key_perm = None
        if key_perm is not None:
            if not isinstance(key_perm, Tensor):
                key_perm = torch.tensor(key_perm, dtype=torch.long, device=self.device)
            self._key_perm = key_perm.to(device=self.device, dtype=torch.long)
        self._host_perm = None
        self._hp = None       # cached ctypes dok_hash_params
        self._bare_plan = None          # of the slot array that `_allocate` made, without hash parameters
        self._plan = None     # what the native calls need to know of this table (_native_plan)
        self._table = None

    # ------------------------------------------------------------------ parameters (lazy, reference order)
    def _current_key_size(self):
        assert self._slots is not None or self._key_size is not None
        if self._slots is not None:
            return math.prod(self._key_shape)
        return int(self._key_size)

    def _draw(self, name):
        """A parameter that the caller did not give, drawn with the reference's calls (:66-113)."""
        ks = self._current_key_size()
        if name == "prime1":
            raw = [np.random.randint(self.n_buckets, self.n_buckets * 2) for _ in range(ks)]
            return [next_prime(r) for r in raw]
        if name == "prime2":
            raw = [np.random.randint(0, 2 ** 60, dtype="int64") for _ in range(ks)]
            return [next_prime(r) for r in raw]
        return [int(np.random.randint(p)) - 1 for p in self._host_param("prime1")]

    def _host_param(self, name):
        values = self._host.get(name)
        if values is None:
            given = self._on_device.get(name)
            values = self._host[name] = self._draw(name) if given is None else given.cpu().tolist()
        return values

    def _param(self, name):
        t = self._on_device.get(name)
        if t is None:
            t = self._on_device[name] = torch.tensor(self._host_param(name), device=self.device, dtype=torch.long)
        return t

    @property
    def prime1(self):
        return self._param("prime1")

    @property
    def prime2(self):
        return self._param("prime2")

    @property
    def alpha1(self):
        return self._param("alpha1")

    @property
    def alpha2(self):
        return self._param("alpha2")

    @property
    def beta1(self):
        return self._param("beta1")

    @property
    def beta2(self):
        return self._param("beta2")

    @property
    def key_perm(self):
        if self._key_perm is None:
            assert self._slots is not None
            self._key_perm = torch.arange(math.prod(self._key_shape), device=self.device)
        else:
            assert self._key_perm.shape[0] == np.prod(self.key_shape)
        return self._key_perm

    @key_perm.setter
    def key_perm(self, new):
        if not isinstance(new, Tensor):
            new = torch.tensor([int(i) for i in new], device=self.device, dtype=torch.long)
        new = new.to(device=self.device, dtype=torch.long)
        assert new.shape == self.key_perm.shape
        self._key_perm = new
        self._host_perm = None
        self._hp = self._plan = None

    def _perm(self):
        """key_perm as host integers."""
        if self._host_perm is None:
            n = math.prod(self._key_shape)
            self._host_perm = list(range(n)) if self._key_perm is None else self._key_perm.cpu().tolist()
            assert len(self._host_perm) == n
        return self._host_perm

    def _materialise_parameters(self):
        # evaluation order of the reference's kernel call (cuda_closed_hashmap.py:350-357)
        if not self._host and not self._on_device:
            # all of them: the four groups below prime1 in one call, which consumes the random state like single ones do
            p = self._host_param("prime1")
            self._host_param("prime2")
            drawn = (np.random.randint(p[0], size=4) if len(p) == 1 else np.random.randint(np.array(p * 4))) - 1
            for i, name in enumerate(_PARAM_NAMES[2:]):
                self._host[name] = drawn[i * len(p):(i + 1) * len(p)].tolist()
        for name in _PARAM_NAMES:
            self._host_param(name)

    # ------------------------------------------------------------------ counters
    @property
    def _state(self):
        if self._counters_of_table is None:
            self._counters_of_table = torch.zeros(_STATE_WORDS, device=self.device, dtype=torch.long)
        return self._counters_of_table

    def _adjust(self, by):
        """n_elements += by (a number or a device scalar) without a change of the slots in use."""
        self._state[_ADJUST] += by
        self._shared.known = False
        self._shared.bound += by if isinstance(by, int) else 0

    def _counter_block(self, block):
        return ctypes.c_void_p(self._state.data_ptr() + 8 * block)

    def _read_state(self):
        return self._state.tolist() if self._plan is None else self._plan.read()

    def _sizes(self, state=None):
        """(n_elements, live slots, tombstones, failed rows) from one read of the counters."""
        c = self._read_state() if state is None else state
        bulk = c[_BY_BULK] + c[_BY_BULK + 1]
        removed = c[_BY_REMOVE + L.CNT_HITS]
        live = c[0] + c[1] + bulk - removed
        # float keys are counted by rows, because their value cast makes different rows share a slot
        inserted = c[_BY_ROWS] if self._key_dtype in L.FLOAT_DTYPES else c[0] + c[1]
        n = inserted + bulk + c[_BY_BULK + L.CNT_HITS] - removed + c[_ADJUST]
        return n, live, removed - c[1], c[L.CNT_FAILED] + c[_BY_BULK + L.CNT_FAILED]

    # ------------------------------------------------------------------ storage
    def _allocate(self, key_shape, key_dtype, value_shape, value_dtype):
        value_bytes = math.prod(value_shape) * value_dtype.itemsize
        key_size = math.prod(key_shape)
        if key_dtype not in L.DTYPE_CODES:
            raise L.DokError(f"unsupported key dtype {key_dtype}")
        if not (1 <= key_size <= L.MAX_KEY_SIZE):
            raise L.DokError(f"keys may have 1..{L.MAX_KEY_SIZE} elements, got {key_size}")
        if not (1 <= value_bytes <= L.MAX_VALUE_BYTES):
            raise L.DokError(f"value rows may have 1..{L.MAX_VALUE_BYTES} bytes, got {value_bytes}")
        self._value_bytes, self._key_bytes = value_bytes, key_size * key_dtype.itemsize
        self._value_shape, self._value_dtype = torch.Size(value_shape), value_dtype
        self._key_shape, self._key_dtype = torch.Size(key_shape), key_dtype
        self._marks = L.native().Marks()
        self._hp = self._plan = None
        device = torch.cuda.current_device() if self.device.index is None else self.device.index
        self._bare_plan, self._slots, self._counters_of_table, layout = L.native().allocate(
            device, self._n_buckets, self._key_shape, key_dtype, self._value_shape, value_dtype, self._counters_of_table)
        self._layout = _Layout(*layout)

    def _begin_bulk_insert(self, key_shape, key_dtype, value_shape, value_dtype, n_new, spare=()):
        """What `set` does to a never-used map before its kernel runs, for a batch known to hold `n_new` pairwise
        different new keys: allocate, draw the parameters, grow if the reference's trigger fires (which re-draws them,
        cuda_closed_hashmap.py:365-366, 456-468).  The caller then inserts the rows with a kernel that counts into
        `_counter_block(_BY_BULK)`.  `spare`: a list of memory that is dropped where there is no room beside it."""
        assert self._slots is None
        if n_new == 0:
            self._allocate(key_shape, key_dtype, value_shape, value_dtype)
            return
        self._key_size = math.prod(key_shape)
        self._materialise_parameters()
        if n_new > int(self._rehash_threshold * self.n_buckets):
            self.__init__(n_buckets=int(n_new * self._rehash_factor), device=self.device, key_perm=self._key_perm,
                          rehash_factor=self._rehash_factor, rehash_threshold=self._rehash_threshold,
                          tombstone_threshold=self._tombstone_threshold)
        try:
            self._allocate(key_shape, key_dtype, value_shape, value_dtype)
        except torch.OutOfMemoryError:
            if not spare:
                raise
            spare.clear()
        if self._slots is None:
            self._allocate(key_shape, key_dtype, value_shape, value_dtype)
        self._materialise_parameters()
        self._shared.exact(n_new)

    def _slot_view(self, dtype, inner_shape, byte_offset):
        """[n_buckets, *inner_shape] strided view of one field of the slot array."""
        es = dtype.itemsize
        strides, acc = [], 1
        for extent in reversed(tuple(inner_shape)):
            strides.append(acc)
            acc *= int(extent)
        strides = (self._layout.slot_bytes // es,) + tuple(reversed(strides))
        return self._slots.view(dtype).as_strided((self._n_buckets,) + tuple(inner_shape), strides, byte_offset // es)

    @property
    def _uuid(self):
        """[n_buckets] int64 tags: uuid, -1 empty, -3 removed (a strided view of the slot array)."""
        if self._slots is None:
            return torch.full((self._n_buckets,), self._empty_marker, device=self.device, dtype=torch.long)
        return self._slot_view(torch.int64, (), 0)

    @property
    def _values(self):
        """[n_buckets, *value_shape] view of the value field of the slots (None before the first set)."""
        if self._slots is None:
            return None
        return self._slot_view(self._value_dtype, self._value_shape, self._layout.value_offset)

    @property
    def _keys(self):
        """[n_buckets, *key_shape] view of the key rows, storage-column order (None before the first set)."""
        if self._slots is None:
            return None
        return self._slot_view(self._key_dtype, self._key_shape, self._layout.key_offset)

    def _next_epoch(self):
        """Epoch of the next stamped set: larger than every epoch stamped on this table before."""
        self._ready_stamps()
        epoch = self._marks.epoch = self._marks.epoch + 1
        return epoch

    def _ready_stamps(self):
        """The stamps live in the slots when the layout has room for them, else in a separate array allocated on first use."""
        marks = self._marks
        if self._layout.stamp_offset < 0 and marks.stamp is None:
            marks.stamp = torch.zeros(self._layout.n_slots, device=self.device, dtype=torch.long)
        if marks.epoch >= L.MAX_EPOCH - 1:
            raise L.DokError("stamp epochs exhausted: rehash() the map to start over")

    def _c_table(self):
        t = L.Table()
        t.slots = self._slots.data_ptr()
        stamp = self._marks.stamp
        t.stamp = stamp.data_ptr() if stamp is not None else None
        t.n_buckets = self._n_buckets
        t.slot_bytes = self._layout.slot_bytes
        t.value_bytes = self._value_bytes
        t.key_bytes = self._key_bytes
        self._table = t   # keeps the struct alive for the duration of the call
        return ctypes.byref(t)

    def _c_hash(self):
        if self._hp is None:
            self._materialise_parameters()
            hp = L.HashParams()
            ks = math.prod(self._key_shape)
            hp.key_size = ks
            hp.key_dtype = L.DTYPE_CODES[self._key_dtype]
            host = self._checked_params()
            for name in _PARAM_NAMES:
                getattr(hp, name)[:ks] = host[name]
            hp.key_perm[:ks] = self._perm()
            self._hp = hp
        return ctypes.byref(self._hp)

    def _checked_params(self):
        ks = math.prod(self._key_shape)
        host = {name: self._host_param(name) for name in _PARAM_NAMES}
        assert all(len(v) == ks for v in host.values())
        assert all(abs(p) >= 2 for p in host["prime1"] + host["prime2"]), "primes must have magnitude >= 2"
        if 0 in host["alpha2"]:
            import warnings
            warnings.warn("alpha2 contains 0: the uuid ignores that key element, so keys differing only there "
                          "are told apart only by their first hash (the reference draws alpha2 from [-1, prime1-2])")
        return host

    def _native_plan(self):
        """The native form of this table, or None where only the general calls serve it."""
        if self._plan is None and self._bare_plan is not None:
            self._materialise_parameters()
            host = self._checked_params()
            self._bare_plan.set_hash(L.DTYPE_CODES[self._key_dtype], host["alpha2"], host["beta2"], host["prime2"], host["alpha1"],
                                     host["beta1"], host["prime1"], self._perm())
            self._plan = self._bare_plan
        elif self._plan is None and self._slots is not None:
            self._c_hash()
            self._c_table()
            self._plan = L.native().Plan(bytes(self._table), bytes(self._hp), self._state.data_ptr(), self._slots.device.index,
                                       tuple(self._key_shape), self._key_dtype, tuple(self._value_shape), self._value_dtype)
        return self._plan

    def _counters(self):
        return torch.zeros(L.N_COUNTERS, device=self.device, dtype=torch.long)

    # The rehash decision of `set` needs n_elements on the host, which the reference gets with a blocking .item()
    # per call.  Here the host keeps an UPPER BOUND instead: every set adds its rows to it, and now and then the device
    # counters are copied to pinned memory without waiting; the bound is then the newest copy that has landed plus the
    # sizes of the batches enqueued after it.  Only when the bound crosses the threshold is the exact value fetched.
    # A copy costs more than a small set, so one is made when the bound has used up a quarter of the room that was left at
    # the last one.
    def _after_mutation(self, added):
        sh = self._shared
        sh.known = False
        sh.bound += added
        for s in sh.snapshots:
            s[1] += added                       # rows that may have been inserted after that snapshot was taken
        room = int(self._rehash_threshold * self._n_buckets) - sh.base
        if 4 * (sh.bound - sh.base) < room:
            return
        if sh.ring is None:
            sh.device = self._slots.device.index
            sh.ring = _rings.take(sh.device)
        in_flight = [s[0] for s in sh.snapshots]
        place = next((i for i in range(8) if i not in in_flight), None)
        if place is None:
            return                              # eight copies still in flight: skip this one, the bound stays valid
        sh.ring.copy(self._native_plan(), place)
        sh.snapshots.append([place, 0])
        sh.base = sh.bound

    def _element_bound(self):
        sh = self._shared
        newest = None
        while sh.snapshots and sh.ring.landed(sh.snapshots[0][0]):
            newest = sh.snapshots.pop(0)
        if newest is not None:
            n = self._sizes(sh.ring.read(newest[0]))[0]
            sh.bound = min(sh.bound, n + newest[1])
            if not sh.snapshots:
                sh.base = min(sh.base, n)
        return sh.bound

    def _room_for(self, rows, limit):
        """bound + rows <= limit?  When the bound is too high only because the host runs ahead of the device, wait
        for the count copies still in flight to land -- oldest first, each an event on the stream -- instead of for the
        whole stream: the device keeps the work that is queued behind them."""
        bound = self._element_bound()
        snaps = self._shared.snapshots
        while bound + rows > limit and snaps:
            self._shared.ring.wait(snaps[0][0])
            bound = self._element_bound()
        return bound + rows <= limit

    # ------------------------------------------------------------------ compaction
    def items(self, keys=True, values=True, uuid=True, transposed_keys=False):
        """(keys, values, uuid) of the live slots in slot order, from one pass over the tags."""
        assert self._slots is not None
        lib = L.lib()
        with L.on(self.device):
            st = L.stream_ptr(self.device)
            tiles = lib.dok_compact_tiles(self._n_buckets)
            offsets = torch.empty(tiles + 1, device=self.device, dtype=torch.long)
            L.check(lib.dok_map_compact_count(self._c_table(), L.ptr(offsets), st), "dok_map_compact_count")
            count = int(offsets[-1].item())
            ks = math.prod(self._key_shape)
            k = v = u = None
            if keys:
                shape = (ks, count) if transposed_keys else (count, ks)
                k = torch.empty(shape, device=self.device, dtype=self._key_dtype)
            if values:
                v = torch.empty((count,) + tuple(self._value_shape), device=self.device, dtype=self._value_dtype)
            if uuid:
                u = torch.empty(count, device=self.device, dtype=torch.long)
            if count:
                L.check(lib.dok_map_compact_scatter(self._c_table(), self._c_hash(), L.ptr(offsets), L.ptr(k),
                                                    int(transposed_keys), L.ptr(v), L.ptr(u), st),
                        "dok_map_compact_scatter")
        return k, v, u

    def count_live(self):
        """Live slots, from the counters that every kernel keeps."""
        return 0 if self._slots is None else self._sizes()[1]

    @property
    def nonempty_mask(self):
        return (self._uuid != self._empty_marker) & (self._uuid != self._removed_marker)

    def keys(self):
        if self._slots is None:
            return None
        return self.items(values=False, uuid=False)[0]

    def values(self):
        if self._slots is None:
            return None
        return self.items(keys=False, uuid=False)[1]

    def uuid(self):
        if self._slots is None:
            return torch.empty(0, device=self.device, dtype=torch.long)
        return self.items(keys=False, values=False)[2]

    def set_values(self, selectors, new_values):
        masked_values = self._values[self.nonempty_mask]
        masked_values[selectors] = new_values
        self._values[self.nonempty_mask] = masked_values

    def permute_keys(self, ordering):
        assert self._slots is not None, "hashmap is empty"
        assert len(self.key_shape) == 1, "keys are not one dimensional"
        assert len(ordering) == self.key_shape[0]
        assert len(set(ordering)) == len(ordering), "duplicates are not allowed"
        self._materialise_parameters()
        self._keys.copy_(self._keys[:, ordering].clone())
        self._host = {name: [self._host_param(name)[i] for i in ordering] for name in _PARAM_NAMES}
        self._on_device = {}
        self._hp = self._plan = None

    def clone(self, deepclone=False):
        self._materialise_parameters()
        cp = (lambda x: x.clone()) if deepclone else (lambda x: x)
        new = CudaClosedHashmap(
            n_buckets=self.n_buckets, device=self.device, **{name: list(self._host_param(name)) for name in _PARAM_NAMES},
            key_perm=None if self._key_perm is None else cp(self._key_perm),
            rehash_factor=self._rehash_factor, rehash_threshold=self._rehash_threshold,
            tombstone_threshold=self._tombstone_threshold,
        )
        if self._slots is None:
            return new           # each will have slots of its own, and whatever goes with them
        new._tombstone_host_bound = self._tombstone_host_bound
        new._slots = cp(self._slots)
        new._layout = self._layout
        new._value_bytes, new._key_bytes = self._value_bytes, self._key_bytes
        new._value_shape, new._value_dtype = self._value_shape, self._value_dtype
        new._key_shape, new._key_dtype = self._key_shape, self._key_dtype
        new._counters_of_table = cp(self._state)
        if deepclone:
            # stamps and numbers in the slots were copied with them: continue; a separate array is copied too
            stamp = self._marks.stamp
            new._marks = L.native().Marks(self._marks, None if stamp is None else stamp.clone())
            new._shared = _Shared(self._shared.bound)
        else:
            new._marks, new._shared = self._marks, self._shared   # a view writes the same slots
        return new

    # ------------------------------------------------------------------ sizes
    @property
    def n_elements(self):
        state = self._read_state()
        n, _, _, failed = self._sizes(state)
        self._shared.exact(n)
        if failed:
            # rows that a set could not store because the table was full (the reference drops them silently,
            # closed_hashmap_impl_class.cu:426; here they are counted and reported where the host synchronises anyway)
            self._state[L.CNT_FAILED] = self._state[_BY_BULK + L.CNT_FAILED] = 0
            raise L.DokError(f"{failed} rows of earlier set calls were not stored: the table was full "
                             f"({self._n_buckets} buckets); rehash() to a larger size and set them again")
        return n

    def _size_on_device(self):
        return torch.tensor(self._sizes()[0], device=self.device)

    @property
    def last_set_failed(self):
        """Rows that set calls could not store so far (table full); reading it synchronises."""
        return self._sizes()[3]

    @property
    def n_buckets(self):
        return self._n_buckets

    @property
    def load_factor(self):
        return self.n_elements / self.n_buckets

    @property
    def n_tombstones(self):
        return int((self._uuid == self._removed_marker).sum().item())

    @property
    def key_shape(self):
        assert self._slots is not None
        return self._key_shape

    @property
    def value_shape(self):
        assert self._slots is not None
        return self._value_shape

    @property
    def key_type(self):
        return self._key_dtype

    @property
    def value_type(self):
        return self._value_dtype

    def __len__(self):
        return self.n_elements

    # ------------------------------------------------------------------ python-side hashes of the reference
    def _keys_as_long_bits(self, keys):
        n_keys = keys.shape[0]
        keys = keys.reshape(n_keys, -1).clone()
        if keys.dtype == torch.float:
            keys = keys.view(dtype=torch.int32).long()
            keys[keys == -2 ** 31] = 0
        elif keys.dtype == torch.half:
            keys = keys.view(dtype=torch.int16).long()
            keys[keys == -2 ** 15] = 0
        elif keys.dtype == torch.double:
            keys = keys.view(dtype=torch.int64)
            keys[keys == -2 ** 63] = 0
        else:
            keys = keys.to(torch.long)
        return keys

    def get_hash(self, keys):
        """Python-side first hash of the reference (cuda_closed_hashmap.py:278-300; bit-casts floats, unlike the
        kernels).  Diagnostic only: this library does not place rows with it."""
        keys = self._keys_as_long_bits(keys)
        terms = (self.alpha1[None] * keys + self.beta1[None]) % self.prime1[None]
        if self._key_perm is not None:
            terms = terms[:, self._key_perm]
        return terms.prod(dim=-1).abs() % self.n_buckets

    def get_uuid(self, keys):
        """Python-side second hash of the reference (cuda_closed_hashmap.py:302-319).  `device_uuid` returns what
        the kernels use."""
        keys = self._keys_as_long_bits(keys)
        return ((self.alpha2[None] * keys + self.beta2[None]) % self.prime2[None]).prod(dim=-1).abs()

    def test_uniformity(self, keys):
        hash_codes = self.get_hash(keys)
        logits = (torch.bincount(hash_codes, minlength=self.n_buckets) + 1).log()
        logp = torch.log_softmax(logits, dim=-1)
        return (-(logp * logp.exp()).sum(dim=-1)).exp() / self.n_buckets

    def device_uuid(self, keys):
        """uuid of each key row exactly as the kernels compute it (value cast of the key elements)."""
        assert self._slots is not None
        keys = keys.contiguous()
        out = torch.empty(keys.shape[0], device=self.device, dtype=torch.long)
        with L.on(self.device):
            L.check(L.lib().dok_map_uuid(self._c_table(), self._c_hash(), L.ptr(keys), keys.shape[0], L.ptr(out), None,
                                         L.stream_ptr(self.device)), "dok_map_uuid")
        return out

    # ------------------------------------------------------------------ set
    def _launch_set(self, keys, values, assume_unique):
        """The set kernels on contiguous rows of this table."""
        plan = self._native_plan()
        if plan.set(keys, values, assume_unique, self._marks) is None:
            self._ready_stamps()
            plan.set(keys, values, assume_unique, self._marks)

    def set(self, new_keys, new_values, assume_unique=False):
        """Insert-or-assign a batch.  `assume_unique=True` promises pairwise different keys and runs one kernel
        instead of two.  Returns None like the reference."""
        plan = self._plan
        if plan is not None and self._key_dtype not in L.FLOAT_DTYPES \
                and self._room_for(new_keys.shape[0], int(self._rehash_threshold * self._n_buckets)):
            rows = plan.set(new_keys, new_values, assume_unique, self._marks)
            if rows is not None:
                self._after_mutation(rows)
                return
        assert new_keys.shape[0] == new_values.shape[0]
        if self._slots is None:
            assert new_keys.device == new_values.device == self.device
            self._allocate(new_keys.shape[1:], new_keys.dtype, new_values.shape[1:], new_values.dtype)
        else:
            assert new_keys.dtype == self._key_dtype
            assert new_keys.device == self.device
            assert new_keys.shape[1:] == self._key_shape
            assert new_values.dtype == self._value_dtype
            assert new_values.device == self.device
            assert new_values.shape[1:] == self._value_shape
        new_keys = new_keys.contiguous()
        new_values = new_values.contiguous()
        n = new_keys.shape[0]
        if n == 0:
            return
        self._materialise_parameters()
        limit = int(self._rehash_threshold * self.n_buckets)
        row_counted = new_keys.dtype in L.FLOAT_DTYPES
        # Where the bound may only be stale (the host runs ahead of the device), the exact count is fetched before paying for
        # a pass that counts the distinct new keys.  These (cuda_closed_hashmap.py:350-363) are counted with a scratch set on
        # the device: uuids of integer keys, ROWS of floating ones like in the reference, because the value cast makes many
        # rows share a uuid.
        plan = self._native_plan()
        if self._room_for(n, limit) or (not self._shared.known and self.n_elements + n <= limit):
            # whatever the number of new keys is, the reference would not rehash: insert and count on the device
            if row_counted:
                plan.count_new(new_keys, _BY_ROWS, False, self._shared.bound == 0)
            self._launch_set(new_keys, new_values, assume_unique)
            self._after_mutation(n)
            return
        state = plan.count_new(new_keys, _COUNTED_NEW, True, self._shared.bound == 0)
        n_elements, live, _, failed = self._sizes(state)
        if failed:
            self.n_elements             # raises
        n_new = state[_COUNTED_NEW]
        if n_elements + n_new > limit:
            self.rehash(int((n_elements + n_new) * self._rehash_factor), live)
        self._launch_set(new_keys, new_values, assume_unique)
        if row_counted:
            self._state[_BY_ROWS] += n_new
        self._shared.exact(n_elements + n_new)

    def set_rows(self, keys, values, assume_unique=False):
        """Kernel only, like `remove_rows`: insert-or-assign without the reference's bookkeeping around it -- no count
        of the distinct new keys, no rehash decision, no host synchronisation.  New slots are counted on the device.
        The caller guarantees room (rows that find the table full are counted in `last_set_failed`)."""
        assert keys.shape[0] == values.shape[0]
        if self._slots is None:
            self._allocate(keys.shape[1:], keys.dtype, values.shape[1:], values.dtype)
        assert keys.dtype == self._key_dtype and keys.shape[1:] == self._key_shape and keys.device == self.device
        assert values.dtype == self._value_dtype and values.shape[1:] == self._value_shape and values.device == self.device
        if keys.shape[0] == 0:
            return
        self._materialise_parameters()
        before = self._slots_claimed()
        self._launch_set(keys.contiguous(), values.contiguous(), assume_unique)
        if keys.dtype in L.FLOAT_DTYPES:
            self._state[_BY_ROWS] += self._slots_claimed() - before
        self._after_mutation(keys.shape[0])

    def _slots_claimed(self):
        """For sets that count the new SLOTS of float keys where `set` counts rows: the slots claimed so far."""
        return self._state[:2].sum() if self._key_dtype in L.FLOAT_DTYPES else None

    # ------------------------------------------------------------------ sliced batches (the inbox of a sharded map)
    # keys / values / outputs hold n_slices * slice_rows rows; only the first counts[s] rows of slice s are in use, and
    # the counts (device int64[n_slices]) are read by the kernels, so nothing here waits for them.  `abort` (device
    # int64[1] or None): non-zero when the kernels run = do nothing.
    def _sliced_check(self, keys, n_slices, slice_rows, counts):
        assert self._slots is not None, "store something first"
        assert keys.dtype == self._key_dtype and keys.device == self.device and keys.is_contiguous()
        assert keys.shape == (n_slices * slice_rows,) + tuple(self._key_shape)
        assert counts.dtype == torch.long and counts.shape == (n_slices,) and counts.is_contiguous()

    def get_sliced(self, keys, n_slices, slice_rows, counts, abort, fallback_value, values, is_found):
        self._sliced_check(keys, n_slices, slice_rows, counts)
        fb, _keep = self._fallback_ptr(fallback_value)
        with L.on(self.device):
            L.check(L.lib().dok_map_get_sliced(self._c_table(), self._c_hash(), L.ptr(keys), n_slices, slice_rows,
                                               L.ptr(counts), L.ptr(abort), L.ptr(values), L.ptr(is_found), fb, None,
                                               L.stream_ptr(self.device)), "dok_map_get_sliced")

    def remove_sliced(self, keys, n_slices, slice_rows, counts, abort, is_removed):
        self._sliced_check(keys, n_slices, slice_rows, counts)
        cnt = self._counter_block(_BY_REMOVE)
        with L.on(self.device):
            L.check(L.lib().dok_map_remove_sliced(self._c_table(), self._c_hash(), L.ptr(keys), n_slices, slice_rows,
                                                  L.ptr(counts), L.ptr(abort), L.ptr(is_removed), cnt,
                                                  L.stream_ptr(self.device)), "dok_map_remove_sliced")
        self._tombstone_host_bound += n_slices * slice_rows
        self._after_mutation(0)

    def set_sliced(self, keys, values, n_slices, slice_rows, counts, abort, assume_unique=False):
        """Insert-or-assign of a sliced batch.  As long as the table cannot reach its rehash threshold even if every
        row of every slice were new, everything stays on the device.  Otherwise the counts are read (a synchronisation
        of this rank only) and the slices go through `set` one after the other, which may rehash."""
        self._sliced_check(keys, n_slices, slice_rows, counts)
        assert values.dtype == self._value_dtype and values.is_contiguous()
        assert values.shape == (n_slices * slice_rows,) + tuple(self._value_shape)
        self._materialise_parameters()
        rows = n_slices * slice_rows
        limit = int(self._rehash_threshold * self.n_buckets)
        if self._room_for(rows, limit) or self.n_elements + rows <= limit:
            with L.on(self.device):
                epoch, scratch, before = 0, None, self._slots_claimed()
                if not assume_unique:
                    epoch = self._next_epoch()
                    scratch = torch.empty(rows + 1, device=self.device, dtype=torch.long)
                L.check(L.lib().dok_map_set_sliced(self._c_table(), self._c_hash(), L.ptr(keys), L.ptr(values), n_slices,
                                                   slice_rows, L.ptr(counts), L.ptr(abort), L.ptr(scratch), epoch,
                                                   int(bool(assume_unique)), self._counter_block(_BY_SET),
                                                   L.stream_ptr(self.device)), "dok_map_set_sliced")
                if before is not None:
                    self._state[_BY_ROWS] += self._slots_claimed() - before
            self._after_mutation(rows)
            return
        if abort is not None and int(abort.item()) != 0:
            return
        for s, c in enumerate(counts.tolist()):
            if c:
                self.set(keys[s * slice_rows:s * slice_rows + c], values[s * slice_rows:s * slice_rows + c],
                         assume_unique=assume_unique)

    def _fallback_ptr(self, fallback_value):
        """-> (host pointer for the C ABI or None, the host tensor that must stay alive for the call)"""
        if fallback_value is None:
            return None, None
        if not isinstance(fallback_value, torch.Tensor):
            fallback_value = torch.tensor(fallback_value, dtype=self._value_dtype)
        host = torch.broadcast_to(fallback_value.to(dtype=self._value_dtype, device="cpu"), self.value_shape).contiguous()
        return ctypes.c_void_p(host.data_ptr()), host

    # ------------------------------------------------------------------ get
    def get(self, keys, fallback_value=None, values=None, is_found=None):
        """`values` / `is_found`: optional preallocated outputs (contiguous, [n, *value_shape] and bool [n]), like the
        `values=` argument of the reference launcher (closed_hashmap_impl.py:63)."""
        if values is None and is_found is None and fallback_value is None:
            plan = self._plan or self._native_plan()
            out = None if plan is None else plan.get(keys)
            if out is not None:
                return out
        if self._slots is None:
            raise RuntimeError("store something first")
        if keys.shape[0] == 0:
            return (torch.empty(0, *self.value_shape, device=self.device, dtype=self._value_dtype),
                    torch.empty(0, device=self.device, dtype=torch.bool))
        assert keys.dtype == self._key_dtype
        assert keys.device == self.device
        assert keys.shape[1:] == self.key_shape
        fb, _keep = self._fallback_ptr(fallback_value)
        keys = keys.contiguous()
        n = keys.shape[0]
        if values is None:
            values = torch.empty(n, *self.value_shape, device=self.device, dtype=self._value_dtype)
        else:
            assert values.dtype == self._value_dtype and values.is_cuda and values.is_contiguous()
            assert values.shape == (n, *self.value_shape)
        if is_found is None:
            is_found = torch.empty(n, device=self.device, dtype=torch.bool)
        else:
            assert is_found.dtype == torch.bool and is_found.shape == (n,) and is_found.is_contiguous()
        with L.on(self.device):
            L.check(L.lib().dok_map_get(self._c_table(), self._c_hash(), L.ptr(keys), n, L.ptr(values), L.ptr(is_found),
                                        fb, None, L.stream_ptr(self.device)), "dok_map_get")
        return values, is_found

    def probe_stats(self, keys):
        """(mean probe length, hit rate) of a lookup batch."""
        keys = keys.contiguous()
        n = keys.shape[0]
        values = torch.empty(n, *self.value_shape, device=self.device, dtype=self._value_dtype)
        cnt = self._counters()
        with L.on(self.device):
            L.check(L.lib().dok_map_get_probe_stats(self._c_table(), self._c_hash(), L.ptr(keys), n, L.ptr(values), None,
                                                    L.ptr(cnt), L.stream_ptr(self.device)), "dok_map_get_probe_stats")
        cnt = cnt.cpu()
        return cnt[L.CNT_PROBES].item() / max(n, 1), cnt[L.CNT_HITS].item() / max(n, 1)

    # ------------------------------------------------------------------ remove
    def remove_rows(self, keys, is_removed=None):
        """Kernel only: flags aligned to the rows given (no dedup, no sort).  Equal rows report once.
        `is_removed`: optional preallocated bool[n] output."""
        if is_removed is None:
            plan = self._plan or self._native_plan()
            out = None if plan is None else plan.remove_rows(keys)
            if out is not None:
                self._account_removal(out.shape[0])
                return out
        keys = keys.contiguous()
        n = keys.shape[0]
        if is_removed is None:
            is_removed = torch.empty(n, device=self.device, dtype=torch.bool)
        else:
            assert is_removed.dtype == torch.bool and is_removed.shape == (n,) and is_removed.is_contiguous()
        with L.on(self.device):
            L.check(L.lib().dok_map_remove(self._c_table(), self._c_hash(), L.ptr(keys), n, L.ptr(is_removed),
                                           self._counter_block(_BY_REMOVE), L.stream_ptr(self.device)), "dok_map_remove")
        self._account_removal(n)
        return is_removed

    def _account_removal(self, rows):
        self._tombstone_host_bound += rows
        self._after_mutation(0)
        self._maintain()

    def _maintain(self):
        """Rebuild in place when live + tombstone slots exceed the tombstone threshold.  The host first looks at its
        own upper bounds (no synchronisation) and reads the device counts only when they cross."""
        if self._tombstone_threshold is None or self._slots is None:
            return
        auto = self._tombstone_threshold == "auto"
        limit = (0.95 if auto else self._tombstone_threshold) * self.n_buckets
        least = max(1, int(0.02 * self.n_buckets)) if auto else 1
        if self._tombstone_host_bound < least or self._element_bound() + self._tombstone_host_bound <= limit:
            return
        n, _, tombstones, _ = self._sizes()
        self._tombstone_host_bound = tombstones
        if tombstones >= least and n + tombstones > limit:
            try:
                self.rebuild()
            except torch.OutOfMemoryError:
                import warnings
                warnings.warn("no room for a second slot array: the table keeps its tombstones "
                              f"({tombstones} of {self.n_buckets} buckets)")
                self._tombstone_host_bound = 0

    def rebuild(self):
        """The same table without its tombstones: a fresh slot array of the same geometry, every live slot re-inserted
        with the SAME hash parameters (one kernel, dok_map_reinsert).  Lookups, sizes and parameters are unchanged;
        shallow clones made before keep the old slot array (as after a rehash in the reference) with its counters and
        marks."""
        if self._slots is None:
            return
        old_slots, old_state, old_stamp = self._slots, self._state, self._marks.stamp
        source = L.Table()
        source.slots = old_slots.data_ptr()
        source.stamp = old_stamp.data_ptr() if old_stamp is not None else None
        source.n_buckets = self._n_buckets
        source.slot_bytes = self._layout.slot_bytes
        source.value_bytes, source.key_bytes = self._value_bytes, self._key_bytes
        fresh = torch.empty(self._layout.total_bytes, device=self.device, dtype=torch.uint8)     # may raise: nothing changed yet
        state = old_state.clone()
        known = self._shared.known
        self._slots, self._counters_of_table, self._marks, self._shared = fresh, state, L.native().Marks(), _Shared(self._shared.bound)
        self._shared.known = known
        self._plan = self._bare_plan = None
        with L.on(self.device):
            st = L.stream_ptr(self.device)
            L.check(L.lib().dok_map_init(self._c_table(), st), "dok_map_init")
            L.check(L.lib().dok_map_reinsert(ctypes.byref(source), self._c_table(), self._c_hash(), None, st),
                    "dok_map_reinsert")
        # the sizes are those of before; only the tombstones are gone: reused = removed
        gone = state[_BY_REMOVE + L.CNT_HITS] - state[L.CNT_REUSED_REMOVED]
        state[L.CNT_CLAIMED_EMPTY] -= gone
        state[L.CNT_REUSED_REMOVED] += gone
        for old in (old_slots, old_state):
            old.record_stream(torch.cuda.current_stream(self.device))
        self._tombstone_host_bound = 0

    @property
    def tombstone_bound(self):
        """Upper bound of the tombstone slots, from the device counters (exact unless DOK assignments reused some)."""
        return self._sizes()[2]

    def remove(self, keys):
        plan = self._plan or self._native_plan()
        out = None if plan is None else plan.remove(keys)
        if out is not None:
            self._account_removal(out.shape[0])
            return out
        if self._slots is None:
            raise RuntimeError("store something first")
        if keys.shape[0] == 0:
            return torch.zeros(0, device=keys.device, dtype=torch.bool)
        assert keys.dtype == self._key_dtype
        assert keys.device == self.device
        assert keys.shape[1:] == self.key_shape
        if math.prod(self._key_shape) == 1 and keys.dtype not in L.FLOAT_DTYPES:
            # one integer column: a flat radix-sort unique gives the rows of `unique(dim=0)` in the same (sorted) order
            # without the lexicographic row sort
            unique_keys = torch.unique(keys.reshape(-1)).reshape((-1,) + tuple(self._key_shape))
        else:
            unique_keys = keys.unique(dim=0)
        return self.remove_rows(unique_keys)

    # ------------------------------------------------------------------ rehash
    def rehash(self, n_buckets, live=None):
        """New table of `n_buckets` with new random parameters holding the live items (cuda_closed_hashmap.py:456-468).
        One kernel walks the old slots and inserts every live one into the new table (dok_map_reinsert): no
        compaction, no pre-get, no unique.  Like the reference's recursive `set`, a table that the live items fill
        beyond the rehash threshold grows once more (and draws its parameters again)."""
        if self._slots is None:
            self.__init__(n_buckets=n_buckets, device=self.device, key_perm=self._key_perm,
                          rehash_factor=self._rehash_factor, rehash_threshold=self._rehash_threshold,
                          tombstone_threshold=self._tombstone_threshold)
            return
        if live is None:
            live = self.count_live()
        old_slots, source = self._slots, self._native_plan() if live else None          # kept alive until the kernel has run
        geometry = (self._key_shape, self._key_dtype, self._value_shape, self._value_dtype)
        self.__init__(
            n_buckets=n_buckets, device=self.device, key_perm=self._key_perm,
            rehash_factor=self._rehash_factor, rehash_threshold=self._rehash_threshold,
            tombstone_threshold=self._tombstone_threshold,
        )
        self._begin_bulk_insert(*geometry, live)
        if live:
            self._native_plan().reinsert(source)
            old_slots.record_stream(torch.cuda.current_stream(self.device))

    # ------------------------------------------------------------------ persistence
    def state_dict(self):
        """Everything needed to rebuild the map, independent of the slot layout: the live (key, value) rows from one
        compaction pass, the hash parameters (so that uuids, and with them the owner shards of a sharded map, stay
        the same) and the sizing options.  Tombstones are not kept.  The reference has no checkpoint format."""
        if self._slots is not None:
            self._materialise_parameters()
        state = {"format": 1, "n_buckets": self.n_buckets, "rehash_factor": self._rehash_factor,
                 "rehash_threshold": self._rehash_threshold, "tombstone_threshold": self._tombstone_threshold,
                 "key_perm": None if self._key_perm is None else self._key_perm.cpu(), "keys": None, "values": None}
        for name in _PARAM_NAMES:
            drawn = name in self._host or name in self._on_device
            state[name] = torch.tensor(self._host_param(name), dtype=torch.long) if drawn else None
        if self._slots is not None:
            keys, values, _ = self.items(uuid=False)
            state["keys"] = keys.reshape((-1,) + tuple(self.key_shape)).cpu()
            state["values"] = values.cpu()
            state["n_elements"] = self.n_elements            # may over-count like the reference's DOK assignments do
        return state

    @classmethod
    def from_state_dict(cls, state, device="cuda:0"):
        assert state.get("format") == 1
        table = cls(n_buckets=state["n_buckets"], device=device, rehash_factor=state["rehash_factor"],
                    rehash_threshold=state["rehash_threshold"], tombstone_threshold=state.get("tombstone_threshold"),
                    key_perm=state["key_perm"],
                    **{name: None if state[name] is None else state[name].tolist() for name in _PARAM_NAMES})
        if state["keys"] is not None:
            keys, values = state["keys"].to(table.device), state["values"].to(table.device)
            if keys.shape[0]:      # items() gives key columns in the caller's order, like rehash relies on
                table.set(keys, values, assume_unique=True)
            else:
                table._allocate(keys.shape[1:], keys.dtype, values.shape[1:], values.dtype)
            table._adjust(int(state["n_elements"]) - table.n_elements)
        return table

    def __getitem__(self, keys):
        return self.get(keys)

    def __setitem__(self, keys, values):
        return self.set(keys, values)

    def __delitem__(self, keys):
        return self.remove(keys)
