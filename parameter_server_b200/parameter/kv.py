"""Push/Pull containers on the device data plane with the reference's calling
conventions: timestamps, ``wait`` dependencies, callbacks and ``wait(ts)``.

:class:`DeviceKVMap` is the device form of ``KVMap`` (``parameter/kv_map.h:32-66``):
the server side keeps a hash table and runs an entry update (FTRL / AdaGrad / SGD
/ plain sum) on every pushed key; :class:`DeviceKVVector` is the ``sum`` flavour
used like ``KVVector`` with ``PLUS`` merging (``parameter/kv_vector.h:171-211``).
Every rank calls ``push`` for every round (possibly with no keys), because the
owner aggregates one round from all live workers -- the device counterpart of
"an empty but valid slice is still sent" (``system/message.h:136-137``).

With ``exchange=True`` (the default) pulls use the two-sided exchange kernel (keys
to the owners in bulk, weights back in bulk), which is what NVLink likes; then
``pull`` is collective as well: every rank calls it for every round, possibly
with no keys. ``exchange=False`` keeps the one-sided pull (remote probes), which
any rank may call on its own.

Values may be ``k`` floats wide (``KVVector<K,V>(buffer_value, k)``,
``parameter/kv_vector.h:43-104``): pushes take and pulls return ``(n, k)`` arrays.
``channels`` independent key/value sets share the object (``kv[chl]`` in the
reference): ``push`` / ``pull`` take a ``channel``. With ``buffer_value=True`` a
push round is not merged into the channel: the owner finds what every worker
sent under :meth:`buffer` (per source, keys and values), and merges it itself
(:meth:`apply_buffer`, or by pushing something else), which is the reference's
aggregation idiom (``kv_vector.h:182-207``, ``test/kv_vector_buffer_ps.cc:10-59``).

Timestamps are per object and increase by one per request unless given.
Requests run in stream order; ``wait=[t]`` makes a request's kernels wait for
the CUDA event of request ``t``, and ``wait(ts)`` blocks the host until request
``ts`` has finished on the device (then runs its callback).
"""
from __future__ import annotations

import weakref
from typing import Callable, Dict, List, Optional

import numpy as np
import torch

from ..ops import _lib
from ..ops.localize import LocalBatch
from ..parallel.dataplane import DataPlane, OptimizerConfig, PlaneConfig, heap_layout
from ..parallel.fabric import Fabric


class DeviceKVMap:
    def __init__(self, plane: DataPlane, max_keys: int = 1 << 20, buffer_value: bool = False):
        self.plane = plane
        self.max_keys = max_keys
        self.k = plane.width
        self.buffer_value = buffer_value
        self._push_round_of: Dict[int, int] = {}      # timestamp -> push round (for buffer())
        self.dev = plane.device
        self._time = -1
        self._round = 0                       # push rounds seen by the owners
        self._pull_round = 0                  # exchange rounds (pulls)
        self._events: Dict[int, torch.cuda.Event] = {}
        self._callbacks: Dict[int, Callable] = {}
        self._results: Dict[int, torch.Tensor] = {}
        self._bufs: List[LocalBatch] = [LocalBatch(1, max_keys, plane.S, self.dev) for _ in range(4)]
        if self.k > 1:
            for b in self._bufs:                      # k values per key, key-major, for programs that fill a buffer themselves
                b.grad = torch.zeros(max_keys * self.k, dtype=torch.float32, device=self.dev)
        self._next_buf = 0
        self.stream = torch.cuda.Stream(device=self.dev)
        # The plane's status word as a pull leaves it, copied behind the pull into a word of its own: its wait() then needs
        # no blocking transfer. (With on_stream and run_behind, and the kernels' tails: push and pull of 1000 keys 133 ->
        # 88 us.) Only the device writes these words, and in stream order, so that a word may go to another pull while a
        # discarded one's copy is still to come; a pull that finds none free is waited for as a push is.
        self._status_host = torch.zeros(64, dtype=torch.int32, pin_memory=True)
        self._status_seen = self._status_host.numpy()
        self._status_free: List[int] = list(range(len(self._status_seen)))
        self._status_word: Dict[int, int] = {}        # timestamp of a pull -> its word
        # The allocator of pinned memory does not know of these copies: a container that is dropped with a pull in flight
        # gives the words back when its stream is idle.
        weakref.finalize(self, self.stream.synchronize).atexit = False

    @classmethod
    def create(cls, fabric_or_none=None, *, table_capacity: int = 1 << 20, max_keys: int = 1 << 18,
               opt: Optional[OptimizerConfig] = None, ring: int = 4, quant: str = "none", world: int = 1,
               exchange: bool = True, key_cache: bool = False, k: int = 1, channels: int = 1,
               buffer_value: bool = False):
        """``fabric_or_none``: an existing fabric whose heap is large enough, or None to
        make one: over the default process group when ``torch.distributed`` is
        initialised with more than one rank, else a single-GPU heap. ``key_cache``
        turns the key-caching filter on: a pull whose key list equals the previous
        pull's sends no keys (decided inside the exchange kernel)."""
        pc = PlaneConfig(table_capacity=table_capacity, inbox_cap=max_keys, ring=ring, quant=quant,
                         pull_cap=max_keys if exchange else 0, key_cache=key_cache, width=k, channels=channels)
        fab = fabric_or_none
        if fab is None:
            import torch.distributed as dist
            if dist.is_available() and dist.is_initialized() and dist.get_world_size() > 1:
                fab = Fabric.from_process_group(heap_layout(pc, dist.get_world_size()).total())
            else:
                fab = Fabric.single(heap_layout(pc, world).total())
        return cls(DataPlane(fab, pc, opt or OptimizerConfig(algo="sum")), max_keys, buffer_value=buffer_value)

    def _stamp(self, ts: Optional[int]) -> int:
        ts = self._time + 1 if ts is None or ts < 0 else ts
        self._time = max(self._time, ts)
        return ts

    def _begin(self, wait: Optional[List[int]]):
        _lib.run_behind(self.stream, torch.cuda.current_stream(self.stream.device.index))
        for t in wait or []:
            ev = self._events.get(t)
            if ev is not None:
                self.stream.wait_event(ev)

    def _release_word(self, ts: int):
        word = self._status_word.pop(ts, None)
        if word is not None:
            self._status_free.append(word)

    def _finish(self, ts: int, callback, word: Optional[int] = None):
        ev = torch.cuda.Event()
        ev.record(self.stream)
        self._release_word(ts)                        # (of an earlier request with this timestamp)
        if word is not None:
            self._status_word[ts] = word
        self._events[ts] = ev
        if callback is not None:
            self._callbacks[ts] = callback

    def _buffer(self, keys: torch.Tensor) -> LocalBatch:
        # A request with the very key tensor of the request before it (the usual push-then-pull pair; same
        # object, not written to since) reuses that request's key buffer and owner offsets: a launch less.
        tag = (id(keys), keys._version, keys.data_ptr(), keys.numel())
        if tag == self.__dict__.get("_last_keys_tag"):
            return self._last_buf
        b = self._bufs[self._next_buf]
        self._next_buf = (self._next_buf + 1) % len(self._bufs)
        keys.record_stream(self.stream)               # read on this stream: its memory stays until then
        b.set_keys(keys, self.plane.bounds, stream=self.stream)
        self._last_keys_tag, self._last_buf, self._last_keys = tag, b, keys      # (keeps the tensor, and so its id, alive)
        return b

    def _in_place(self, values) -> bool:
        """Whether the push kernel, which reads adjacent floats from one address, can read ``values`` where it is."""
        return (isinstance(values, torch.Tensor) and values.is_cuda and values.dtype == torch.float32
                and values.is_contiguous() and not values.is_neg() and values.device == self.stream.device)

    def _ready(self, k: torch.Tensor, values) -> bool:
        """Whether a push need not enter the container's stream: no conversion is to run there, and its device is the
        current one already (launches go to the current device, whatever their stream)."""
        return (self._in_place(values) and k.dtype == torch.int64 and k.is_contiguous() and k.device == values.device
                and torch.cuda.current_device() == self.stream.device.index)

    @staticmethod
    def _as_keys(keys, dev) -> torch.Tensor:
        if isinstance(keys, torch.Tensor):
            return keys.to(dev)
        k = np.ascontiguousarray(np.asarray(keys, dtype=np.uint64))
        assert (np.diff(k.astype(np.float64)) > 0).all() if len(k) > 1 else True, "keys must be sorted and unique"
        return torch.from_numpy(k.view(np.int64)).to(dev)

    def push(self, keys, values, ts: Optional[int] = None, wait: Optional[List[int]] = None, callback=None,
             channel: int = 0) -> int:
        """Push sorted unique uint64 keys with one value (``k`` values: an ``(n, k)`` array) each into
        ``channel``; returns the timestamp. ``values`` on this device is read where it is, on the container's
        stream: leave it unchanged until the request has finished (:meth:`wait`). Both halves of the round
        are enqueued here: the worker half (values into the owners' inboxes) and this rank's owner half
        (merge of the round)."""
        ts = self._stamp(ts)
        self._begin(wait)
        k = self._as_keys(keys, self.dev)
        with _lib.on_stream(None if self._ready(k, values) else self.stream):
            rnd = self._push_round_of[ts] = self._push_half(k, values)
            self._apply_half(rnd, channel)
        self._finish(ts, callback)
        return ts

    def push_only(self, keys, values) -> int:
        """The worker half of a push round: the values go into the owners' inboxes. Returns the round.
        The owner half is :meth:`apply_round`; :meth:`push` does both, the node-level customers
        (``parameter/kv_nodes.py``) let the server node decide when the round is merged. There is no
        request to wait for: ``values`` is read in the order of the caller's current stream, which may
        write to it again right after the call."""
        if isinstance(values, torch.Tensor) and values.device.type == torch.device(self.dev).type:
            values = values.clone()                   # (from the host the copy to the device is a private one)
        k = self._as_keys(keys, self.dev)
        self._begin(None)
        with torch.cuda.stream(self.stream):
            return self._push_half(k, values)

    def _push_half(self, k: torch.Tensor, values) -> int:
        """The worker half of a round, on this container's stream (which is the current one where ``values`` or ``k`` are
        still to be converted)."""
        b = self._buffer(k)
        n = k.numel()
        v = None
        if n:
            if isinstance(values, torch.Tensor) and values.is_cuda:
                values.record_stream(self.stream)     # read on this stream: its memory stays until then
            # the kernel reads n * k adjacent floats: a column, a step slice or an expanded tensor (which flatten()
            # returns as the strided view that it is) is copied first
            v = values if self._in_place(values) else \
                torch.as_tensor(values, dtype=torch.float32).to(self.dev).flatten().contiguous().resolve_neg()
            assert v.numel() == n * self.k, f"{n} keys of width {self.k} need {n * self.k} values"
        rnd = self._round
        self._round += 1
        self.plane.push(b, rnd, with_gradient=False, values=v, stream=self.stream)
        return rnd

    def apply_round(self, rnd: int, channel: int = 0):
        """The owner half of push round ``rnd``: merge what every live worker sent (a buffered container
        only consumes the round: its ring slot becomes reusable later, the values stay unmerged)."""
        with torch.cuda.stream(self.stream):
            self._apply_half(rnd, channel)

    def _apply_half(self, rnd: int, channel: int):
        self.plane.apply(rnd, channel=channel, stream=self.stream,
                         opt=OptimizerConfig(algo="keep") if self.buffer_value else None)

    def buffer(self, ts: int):
        """What this rank, as an owner, received in the push with timestamp ``ts``: one
        ``(keys uint64 array, values tensor (n, k))`` pair per source rank. Readable until ``ring - 1``
        further rounds have been pushed (the inbox slot is then reused)."""
        self.wait(ts) if ts in self._events else None
        rnd = self._push_round_of[ts]
        p = self.plane
        q = rnd % p.cfg.ring
        torch.cuda.current_stream(self.dev).synchronize()
        out = []
        for r in range(p.S):
            word = 8 + p.cfg.ring * p.S + q * p.S + r
            n = int(p.ctrl[word].item())
            ko = p.layout["inbox_keys"] + ((q * p.S + r) * p.cfg.inbox_cap) * 8
            vo = p.layout["inbox_vals"] + ((q * p.S + r) * p.cfg.inbox_cap) * 4 * self.k
            keys = p.fabric.view(ko, (n,), torch.int64).cpu().numpy().view(np.uint64)
            vals = p.fabric.view(vo, (n * self.k,), torch.float32).clone().view(n, self.k)
            out.append((keys, vals))
        return out

    def apply_buffer(self, ts: int, channel: int = 0):
        """Merge the buffered round ``ts`` into ``channel`` (sum over the workers, added to the stored values)."""
        rnd = self._push_round_of[ts]
        with torch.cuda.stream(self.stream):
            self.plane.apply(rnd, channel=channel, stream=self.stream, opt=OptimizerConfig(algo="sum"))

    def pull(self, keys, ts: Optional[int] = None, wait: Optional[List[int]] = None, callback=None,
             channel: int = 0) -> int:
        """Pull the values of ``keys`` from ``channel``; the result is available from :meth:`result` after :meth:`wait`."""
        ts = self._stamp(ts)
        k = self._as_keys(keys, self.dev)
        self._begin(wait)
        with _lib.on_stream(self.stream):
            b = self._buffer(k)
            # the owners must have applied every round pushed so far
            if self.plane.cfg.pull_cap:
                rnd = self._pull_round
                self._pull_round += 1
                # one rank: the kernel writes the result; several: the owners write into the response buffer
                n = k.numel()
                out = torch.empty((n, self.k) if self.k > 1 else n, dtype=torch.float32, device=self.dev) if self.plane.S == 1 and n else None
                self.plane.pull_exchange(b, rnd, need_applied=self._round, with_margins=False, channel=channel,
                                         out=out, stream=self.stream)
                self._results[ts] = out if out is not None else self.plane.response_weights(rnd, n).clone()
            else:
                self.plane.pull_margin(b, need_applied=self._round, with_margins=False, stream=self.stream)
                self._results[ts] = b.w_local[:k.numel()].clone()
        word = self._status_free.pop() if self._status_free else None
        if word is not None:
            _lib.check(_lib.lib().psb_read_word(self._status_host.data_ptr() + 4 * word, self.plane.status.data_ptr(),
                                                self.stream.cuda_stream), "status", kernels=0)
        self._finish(ts, callback, word)
        return ts

    def wait(self, ts: int):
        ev = self._events.pop(ts, None)
        if ev is not None:
            ev.synchronize()
        word = self._status_word.get(ts)
        good = ev is not None and word is not None and self._status_seen[word] == 0
        self._release_word(ts)
        if not good:
            self.plane.check_status("kv")
        cb = self._callbacks.pop(ts, None)
        if cb is not None:
            cb()

    def result(self, ts: int) -> torch.Tensor:
        return self._results.pop(ts)

    def discard(self, ts: int):
        """Forget request ``ts`` (its event, callback and pulled values) without waiting for it."""
        self._events.pop(ts, None)
        self._callbacks.pop(ts, None)
        self._results.pop(ts, None)
        self._release_word(ts)

    def write_to_file(self, path: str):
        """``key<TAB>value`` per non-zero entry of this shard."""
        from ..app.linear import write_model
        keys, w = self.plane.dump_nonzero()
        write_model(path, keys.numpy(), w.numpy())


class DeviceKVVector(DeviceKVMap):
    """``sum`` entries: a push adds into the stored values (KVVector PLUS semantics)."""

    @classmethod
    def create(cls, fabric_or_none=None, **kw):
        kw.setdefault("opt", OptimizerConfig(algo="sum"))
        return super().create(fabric_or_none, **kw)
