"""`CudaBackend`: the device backend behind the op interface, standing in for `WebGPUBackend`
(src/backend/webgpu.ts). Same public surface: `install/uninstall`, the 14 ops of `OpsBackend`, the
`RegionBackend` trio, `uploadParams`, `sync`, `reclaimStepTransients`, `residentBytes`, the raw-buffer
calls the optimizers and checkpoints use, and the introspection fields its tests read. Every method
is a thin enqueue through the C ABI of libgguftrain_cuda.so; nothing here computes.

Differences that are deliberate:
 * Gradient buffers are not cleared and then `+=`-ed into. Each entry tracks whether its gradient
   has been written in the current graph; the first writer overwrites, later ones accumulate. The
   values are the ones a cleared buffer plus `+=` would hold, without the clear's memory traffic.
   `gradClearsIssued` counts only the clears that still happen (a gradient that is read before
   anything was written to it, the scatter-add target of the embedding).
 * Work can be captured once into a CUDA graph and replayed (`beginCapture/endCapture`), which is
   what removes the per-op host cost the reference is bound by.
 * `setBatch(B, T)` lets one call carry B sequences as [B*T] rows.
"""
from __future__ import annotations

import ctypes as C
import itertools
from functools import partial
import weakref
from typing import Dict, List, Optional, Sequence

import numpy as np

from . import _lib
from . import autograd as ag
from .autograd import Tensor

_EW = {"add": 0, "mul": 1, "silu": 2, "gelu": 3, "scale": 4}
_KIND = {"NT": 0, "NN": 1, "TN": 2}
PRECISION = {"fp32": 0, "tf32": 1}   # (the C ABI reserves 2 for BF16 and refuses it: there are no BF16 kernels)


_I32 = [None] + [C.c_int32 * n for n in range(1, 9)]     # argument arrays of the grouped launches
_U64 = [None] + [C.c_uint64 * n for n in range(1, 9)]


class _Entry:
    __slots__ = ("owner", "needs", "region", "data", "grad", "bytes", "external", "gradLive", "size", "pendingDx", "copyFrom", "pendingDw", "pendingFwd",
                 "lazy", "ropeOf", "ropeFused", "touched")

    # owner      `_uid` of the backend
    # data       device address; `bytes` long, `size` elements
    # grad       0 for a frozen external (webgpu.ts frozenGradStub), and for an op's output until written
    # needs      an op's output: does a gradient flow through it? (an external: does it have a buffer)
    # region     the recompute region it was made in (0: none): how long a gradient buffer must live
    # touched    an external listed in _touched
    # gradLive   has anything been written to grad in the current graph?
    # pendingDx  (rows, cols, [(dY address, W address, K)]): input-gradient products not launched yet
    # copyFrom   address whose contents are this gradient's value so far (a copy not made yet)
    # pendingDw  a weight-gradient product into this gradient is noted in _pendingDw, not launched yet
    # pendingFwd the projection that produces this tensor is noted in _pendingFwd, not launched yet
    # lazy       a launch that fills `data`: set on a projection (or per-head norm) whose only reader took it rotated, so that it
    #            was never written; run if someone else asks for it (_materializeLazy)
    # ropeOf     for a rotary embedding's output: (input tensor, its entry, H, hd, base, posOffset)
    # ropeFused  its gradient went straight to the rotation's input (attention backward applied it)


_entry = ag.slotMaker(_Entry, dict(grad=0, needs=False, region=0, external=False, touched=False, gradLive=False, pendingDx=None, copyFrom=0,
                                   pendingDw=False, pendingFwd=False, lazy=None, ropeOf=None, ropeFused=False),
                      ("owner", "data", "bytes", "size"))


class CapturedGraph:
    """One recorded stretch of device work, replayable with new integer inputs."""

    def __init__(self, gpu: "CudaBackend", handle: int, inputs, owned, outputs, earlier=()):
        self.gpu = gpu
        self.handle = handle
        self.handles = list(earlier) + [handle]   # segments in order when the recording was cut (cutCapture)
        self.inputs = inputs      # [(addr, count, role, bound)] in upload order
        self.owned = owned        # [(addr, size)] transients pinned to this graph
        self.outputs = outputs    # {name: (addr, count)}

    def writeInputs(self, inputs: Sequence[np.ndarray]):
        """Validate and upload the integer inputs of the next replay. The recorded kernels index the embedding table
        and the logits with these values and have no bound of their own, so the checks the eager ops run above the
        dispatch (assertIdsInTable, keptRowsInVocab: src/model/autograd.ts:813-823, 875-894) run here too."""
        if len(inputs) != len(self.inputs):
            raise ValueError(f"graph takes {len(self.inputs)} integer inputs, got {len(inputs)}")
        g = self.gpu
        staged = []
        for (addr, count, role, bound), arr in zip(self.inputs, inputs):
            if np.asarray(arr).size != count:
                raise ValueError(f"graph input has {np.asarray(arr).size} elements, recorded {count}")
            _checkIntegerInput(arr, role, bound)
            staged.append((addr, _as_u32(arr)))
        for addr, a in staged:
            g._check(g.lib.gt_write(g.ctx, addr, a.ctypes.data, a.nbytes))

    def launch(self, inputs: Sequence[np.ndarray]):
        self.writeInputs(inputs)
        self.replay()

    def replay(self, between=None):
        """Launch the recorded segments in order with the inputs already in place. `between[i]` (if given) is called
        after segment i has been enqueued: host-issued work that cannot be recorded, e.g. a collective."""
        g = self.gpu
        for i, h in enumerate(self.handles):
            g._check(g.lib.gt_graph_launch(g.ctx, h))
            if between is not None and i < len(between) and between[i] is not None:
                between[i]()

    def destroy(self):
        g = self.gpu
        for h in self.handles:
            g._check(g.lib.gt_graph_destroy(g.ctx, h))
        for addr, size in self.owned:
            g._release(addr, size)
        self.owned = []


def _checkIntegerInput(values, role: str, bound: int):
    """The range check of one replayed integer input: `ids` index a table of `bound` rows; `targets` are -1 or a
    vocabulary row; `teacher` ids are vocabulary rows except for a -1 in a row's first slot (checked per element here
    as -1 or a row, the eager op checks the slot rule)."""
    if role is None:
        return
    a = np.asarray(values)
    if a.dtype == np.uint32:
        a = a.astype(np.int64)
        a[a == 0xFFFFFFFF] = -1
    if role == "ids":
        ag.assertIdsInTable(a, bound, "embedding (replay)")
    else:
        bad = np.nonzero((a < -1) | (a >= bound))[0]
        if bad.size:
            t = int(bad[0])
            raise ValueError(f"{role} (replay): value {int(a[t])} at position {t} is not -1 (ignore) or an integer in [0,{bound})")


def _as_u32(values) -> np.ndarray:
    """-1 uploads as 0xffffffff, the marker the kernels test for (webgpu.ts:1636-1646)."""
    a = np.asarray(values)
    if a.dtype != np.uint32:
        a = a.astype(np.int64).astype(np.uint32) if a.dtype.kind != "u" else a.astype(np.uint32)
    return np.ascontiguousarray(a)


class _ProfilingLib:
    """Stand-in for the library handle while a profile is open: every enqueueing call is bracketed by two
    events on the library's stream and attributed to its entry point (and, for products, its layout and
    shape), the per-label GPU time the reference collects with timestamp queries (webgpu.ts:817-880)."""

    _SKIP = ("gt_event_", "gt_read", "gt_write", "gt_sync", "gt_alloc", "gt_free", "gt_stats", "gt_last_error",
             "gt_graph_", "gt_set_", "gt_device_name", "gt_adamw_state", "gt_muon_state", "gt_adamw_get_t",
             "gt_adamw_set_", "gt_muon_set_", "gt_adamw_create", "gt_muon_create", "gt_dp_")

    def __init__(self, lib, ctx, totals):
        self._lib, self._ctx, self._totals = lib, ctx, totals

    def __getattr__(self, name):
        fn = getattr(self._lib, name)
        if name.startswith(self._SKIP):
            return fn
        lib, ctx, totals = self._lib, self._ctx, self._totals

        def timed(*args):
            lib.gt_event_record(ctx, 62)
            st = fn(*args)
            lib.gt_event_record(ctx, 63)
            ms = C.c_float()
            lib.gt_event_elapsed_ms(ctx, 62, 63, C.byref(ms))
            label = name
            if name == "gt_gemm":
                label = f"gt_gemm {('NT', 'NN', 'TN')[args[1]]} {args[3]}x{args[4]}x{args[5]}"
            t = totals.setdefault(label, [0.0, 0])
            t[0] += float(ms.value)
            t[1] += 1
            return st

        return timed


class _Entries:
    """`backend._entries[tensor]`: the device entry of a tensor."""

    __slots__ = ("_gpu",)

    def __init__(self, gpu):
        self._gpu = gpu

    def get(self, t):
        return self._gpu._find(t)

    def __getitem__(self, t):
        e = self._gpu._find(t)
        if e is None:
            raise KeyError(t)
        return e

    def __contains__(self, t):
        return self._gpu._find(t) is not None


_uids = itertools.count(1)


class CudaBackend:
    def __init__(self, device: int = 0, precision: str = "fp32"):
        self.lib = _lib.load()
        ctx = C.c_void_p()
        st = self.lib.gt_init(device, C.byref(ctx))
        if st != 0:
            raise _lib.GtError(st, self.lib.gt_last_error(None).decode())
        self.ctx = ctx
        self.device = device
        name = C.create_string_buffer(256)
        self._check(self.lib.gt_device_name(self.ctx, name, 256))
        self.adapterName = name.value.decode()
        self.timestampSupported = True
        self.lastSyncReadbackBytes = 0
        self.gradClearsIssued = 0
        self.precision = precision
        self._check(self.lib.gt_set_precision(self.ctx, PRECISION[precision]))
        # A tensor's entry sits on the tensor (`Tensor._dev`). Parameters and other externals are listed here as well, so that a
        # tensor two backends take turns with keeps its buffers in both.
        self._uid = next(_uids)
        self._externals: "weakref.WeakKeyDictionary[Tensor, _Entry]" = weakref.WeakKeyDictionary()
        self._tape: List[Tensor] = []          # outputs recorded with a backward closure since the last sync
        self._free: Dict[int, List[int]] = {}  # recycled blocks by size (a dictionary access instead of two library calls)
        self._touched: List[Tensor] = []       # externals used since the last sync
        self._keptOnDevice: "weakref.WeakSet[Tensor]" = weakref.WeakSet()
        self._transients: List[tuple] = []     # (addr, size)
        self._regionFree: List[tuple] = []
        self._outer: List[tuple] = []          # gradient buffers made inside a region for tensors that outlive it
        self._outerMark = 0
        self._regionStack: List[tuple] = []    # (serial of the region, tape length when it opened)
        self._regionsOpened = 0
        # Attention outputs kept across a recompute region (see regionToken / replayOf)
        self.keepAttentionAcrossRecompute = True
        self._regionDepth = 0
        self._curRec: Optional[dict] = None
        self._regionRecs: Dict[int, dict] = {}
        self._nextRegionId = 1
        self._backwardBegun = False
        self._graphSynced = False              # a sync() ran after the current graph was built
        self._graphOpen = False                # forward ops were recorded since the last sync()
        self._capturing = False
        self._captureInputs: List[tuple] = []
        self._captureSegments: List[int] = []
        self._captureMark = 0
        self._batch = (0, 0)
        self._stateBufs: Dict[int, int] = {}
        self._readback = 0
        self._seedBuf = 0
        self._pendingAct = {}   # id(tensor) -> (tensor, op code, input tensor): activations not launched yet
        self._pendingDx: Dict[int, _Entry] = {}   # entries whose gradient still lacks deferred dY.W products
        self.mergeInputGradients = True
        self._pendingFwd: List[dict] = []   # projections of one input not launched yet (see _deferLinear)
        self.groupForward = True
        self._pendingDw: List[tuple] = []   # weight-gradient products not launched yet (see _deferDw)
        self._pendingDwRows = 0
        self.groupWeightGradients = True
        self._pendingAdd = {}   # id(tensor) -> (tensor, a, b): residual adds not launched yet (see add)
        self._pendingCopy: Dict[int, _Entry] = {}  # entries whose gradient is still a view of another buffer (see add)
        self.fuseResidualNorm = True
        self.fuseGatedUnits = True
        self.fuseRope = True               # rotary embeddings applied by the launches before and after them (see rope, attention)
        self.fuseLora = True               # adapter-carrying projections as one op (loraLinear) instead of four
        self._finalizer = weakref.finalize(self, _destroy_ctx, self.lib, self.ctx)

    # ------------------------------------------------------------------ plumbing
    def _check(self, status: int):
        if status != 0:
            raise _lib.GtError(status, self.lib.gt_last_error(self.ctx).decode())

    def describeDevice(self) -> str:
        return self.adapterName

    def startProfile(self):
        """webgpu.ts:817-845. Per-label GPU time until stopProfile(); each call is synchronised, so use it to
        see where time goes, not to measure throughput."""
        if getattr(self, "_profTotals", None) is not None:
            return
        self._profTotals = {}
        self._realLib = self.lib
        self.lib = _ProfilingLib(self._realLib, self.ctx, self._profTotals)

    def stopProfile(self):
        """Returns {label: {"ms": total, "count": n}} and closes the profile (webgpu.ts:847-880)."""
        totals = getattr(self, "_profTotals", None)
        if totals is None:
            return {}
        self.lib = self._realLib
        self._profTotals = None
        return {k: {"ms": v[0], "count": v[1]} for k, v in totals.items()}

    def install(self):
        ag.setOpsBackend(self)

    def uninstall(self):
        ag.setOpsBackend(None)

    def destroy(self):
        """webgpu.ts:764-767."""
        if ag.opsBackend() is self:
            self.uninstall()
        if self._finalizer.alive:
            self._finalizer()
        self.ctx = None

    def setPrecision(self, precision: str):
        self._check(self.lib.gt_set_precision(self.ctx, PRECISION[precision]))
        self.precision = precision

    def setBatch(self, batch: int, seq_len: int = 0):
        """Rows passed to the ops are `batch` sequences of `seq_len` rows; 0 restores one sequence per call."""
        self._check(self.lib.gt_set_batch(self.ctx, batch, seq_len))
        self._batch = (batch, seq_len if batch else 0)

    def stats(self):
        out = (C.c_uint64 * 4)()
        self._check(self.lib.gt_stats(self.ctx, out))
        return {"pool": int(out[0]), "state": int(out[1]), "readback": int(out[2]), "launches": int(out[3])}

    def residentBytes(self):
        """webgpu.ts:774-777."""
        s = self.stats()
        return {"pool": s["pool"], "state": s["state"], "total": s["pool"] + s["state"]}

    def kernelLaunches(self) -> int:
        return self.stats()["launches"]

    @property
    def _entries(self) -> _Entries:
        return _Entries(self)

    # ------------------------------------------------------------------ memory
    def _alloc(self, nbytes: int) -> tuple:
        size = (nbytes + 255) & ~255 if nbytes > 256 else 256
        blocks = self._free.get(size)
        if blocks:
            return blocks.pop(), size
        out = C.c_uint64()
        self._check(self.lib.gt_alloc(self.ctx, size, C.byref(out)))
        return out.value, size

    def _release(self, addr: int, size: int):
        """Back to the pool. One stream: whoever gets the block next is queued behind its last reader."""
        blocks = self._free.get(size)
        if blocks is None:
            self._free[size] = [addr]
        else:
            blocks.append(addr)

    def _acquirePersistent(self, nbytes: int) -> int:
        return self._alloc(nbytes)[0]

    def _acquireTransient(self, nbytes: int) -> int:
        tr = self._alloc(nbytes)
        self._transients.append(tr)
        return tr[0]

    def _acquireRecycled(self, nbytes: int) -> int:
        """Best fit from the region free-list, else a fresh transient (webgpu.ts acquireRecycled)."""
        if not self._regionFree:
            tr = self._alloc(nbytes)
            self._transients.append(tr)
            return tr[0]
        want = (nbytes + 255) & ~255 if nbytes > 256 else 256
        best, bestSize = -1, 0
        for i, (_a, size) in enumerate(self._regionFree):
            if size == want:
                best = i
                break
            if size > want and (best < 0 or size < bestSize):
                best, bestSize = i, size
        if best < 0:
            return self._acquireTransient(nbytes)
        tr = self._regionFree.pop(best)
        self._transients.append(tr)
        return tr[0]

    def _gradAddr(self, e: _Entry) -> int:
        """The gradient buffer of an op's output, made when something is about to be written there: a forward that nothing
        is trained on never has any. One made inside a recompute region for a tensor from outside it outlives the region."""
        if e.grad == 0 and not e.external:
            if e.region == (self._regionStack[-1][0] if self._regionStack else 0):
                e.grad = self._acquireRecycled(e.bytes)
            else:
                tr = self._alloc(e.bytes)
                self._outer.append(tr)
                e.grad = tr[0]
        return e.grad

    def _write(self, addr: int, arr: np.ndarray):
        arr = np.ascontiguousarray(arr)
        self._check(self.lib.gt_write(self.ctx, addr, arr.ctypes.data, arr.nbytes))

    def _read(self, addr: int, out: np.ndarray):
        assert out.flags["C_CONTIGUOUS"]
        if not self._capturing:
            self._flushAllDx("keep")    # whatever is read must not be missing a launch that was put off
        self._check(self.lib.gt_read(self.ctx, addr, out.ctypes.data, out.nbytes))
        self._readback += out.nbytes

    def _readMany(self, wanted):
        """[(address, host array)] as one read."""
        n = len(wanted)
        many = getattr(self.lib, "gt_read_many", None)      # (a stand-in for the library need not have it)
        if n < 2 or many is None:
            for addr, out in wanted:
                self._read(addr, out)
            return
        assert all(a.flags["C_CONTIGUOUS"] for _addr, a in wanted)
        nbytes = [a.nbytes for _addr, a in wanted]
        self._check(many(self.ctx, n, (C.c_uint64 * n)(*[addr for addr, _a in wanted]), (C.c_void_p * n)(*[a.ctypes.data for _addr, a in wanted]),
                         (C.c_uint64 * n)(*nbytes)))
        self._readback += sum(nbytes)

    def _uploadU32(self, values, role: Optional[str] = None, bound: int = 0) -> int:
        if hasattr(values, "addr") and hasattr(values, "bound"):
            return int(values.addr)          # already on the device (ingest.DeviceInts): nothing to upload or replay-patch
        a = _as_u32(values)
        if self._capturing:
            # a replayed graph reads its integer inputs from fixed buffers the launcher rewrites; `role` and `bound`
            # are what the launcher checks new values against
            addr = self._acquirePersistent(a.nbytes)
            self._captureInputs.append((addr, a.size, role, bound))
            return addr
        addr = self._acquireTransient(a.nbytes)
        self._write(addr, a)
        return addr

    def _uploadF32(self, values) -> int:
        a = np.ascontiguousarray(np.asarray(values, dtype=np.float32))
        if self._capturing:
            raise _lib.GtError(4, "float uploads are not replayable; this op cannot be captured")
        addr = self._acquireTransient(a.nbytes)
        self._write(addr, a)
        return addr

    def _find(self, t: Tensor) -> Optional[_Entry]:
        e = t._dev
        if e is None or e.owner == self._uid:
            return e
        return self._externals.get(t)

    def _newExternal(self, t: Tensor, data: int, grad: int) -> _Entry:
        e = _entry(self._uid, data, t.size * 4, t.size)
        e.grad, e.needs, e.external = grad, grad != 0, True
        self._externals[t] = e
        t._dev = e
        return e

    def _entryFor(self, t: Tensor) -> _Entry:
        """webgpu.ts:1539-1573: externals (params, test inputs) get persistent buffers on first use."""
        e = t._dev
        if e is None or e.owner != self._uid:
            e = self._firstUse(t)
        if e.pendingFwd:
            self._flushFwd()
        if e.lazy is not None:
            self._materializeLazy(e)
        if e.external and not e.touched:
            e.touched = True
            self._touched.append(t)
        return e

    def _firstUse(self, t: Tensor) -> _Entry:
        if id(t) in self._pendingAct:
            return self._materializeAct(t)
        if id(t) in self._pendingAdd:
            return self._materializeAdd(t)
        e = self._find(t)
        if e is None:
            if self._capturing:
                raise _lib.GtError(4, "a tensor first reached the device inside a graph capture; upload it first")
            nbytes = t.size * 4
            e = self._newExternal(t, self._acquirePersistent(nbytes), self._acquirePersistent(nbytes) if t.requiresGrad else 0)
            self._write(e.data, t.data)
        return e

    def _entryOf(self, t: Tensor):
        """The device entry of a tensor some op produced (launching it first if it is a deferred activation), or None."""
        e = self._find(t)
        if e is None and id(t) in self._pendingAct:
            e = self._materializeAct(t)
        if e is None and id(t) in self._pendingAdd:
            e = self._materializeAdd(t)
        if e is not None and e.pendingFwd:
            self._flushFwd()
        if e is not None and e.lazy is not None:
            self._materializeLazy(e)
        return e

    @staticmethod
    def _flows(t: Tensor, e: _Entry) -> bool:
        """Does a gradient of `t` have anywhere to go (webgpu.ts:898-901: a frozen input is skipped)?"""
        return e.needs and (t.requiresGrad or not e.external)

    def _makeOut(self, shape: List[int], size: int, prev: List[Tensor], needs: bool) -> tuple:
        t = Tensor.output(shape, size, prev)
        return t, self._newEntry(t, needs)

    def _newEntry(self, t: Tensor, needs: bool) -> _Entry:
        nbytes = t.size * 4
        # (_acquireRecycled written out: this runs once per op)
        blocks = self._free.get((nbytes + 255) & ~255 if nbytes > 256 else 256) if not self._regionFree else None
        if blocks:
            addr = blocks.pop()
            self._transients.append((addr, (nbytes + 255) & ~255 if nbytes > 256 else 256))
        else:
            addr = self._acquireRecycled(nbytes)
        t._dev = e = _entry(self._uid, addr, nbytes, t.size)
        if needs:
            e.needs = t._needs = True
        if self._regionStack:
            e.region = self._regionStack[-1][0]
        return e

    def _record(self, t: Tensor, needs: bool, bw, *args) -> Tensor:
        """Put an op's backward on the tape, or nothing where no gradient can flow: such a tensor is freed with its last reader
        instead of being kept (with everything it was computed from) until the graph goes."""
        if needs:
            t._backward = partial(bw, *args) if args else bw
            self._tape.append(t)
        else:
            t._backward = self._ensureBackwardBegun
            t._prev = []
        return t

    def _dropTape(self, mark: int = 0, keep: Sequence[Tensor] = ()):
        """The buffers of these graphs have been recycled: a backward over them is refused or does nothing, and without their
        closures the tensors are freed by reference count (a closure and its tensor refer to each other, and waiting for the
        cycle collector costs a training loop more time than its launches)."""
        for t in self._tape[mark:]:
            if any(t is k for k in keep):
                continue
            t._backward = self._ensureBackwardBegun
            t._prev = []
        del self._tape[mark:]

    # The input gradient of `linear` is dX (+)= dY.W. An activation that feeds several projections (the normed input
    # of q, k and v; of gate and up) collects one such product per consumer, and the reference issues them one by one,
    # each re-reading and re-writing the [T, in] buffer (src/backend/webgpu.ts:884-903). Here a closure only notes its
    # (dY, W, K); the products are launched together, as one matrix product whose contraction runs over all the K
    # ranges (gt_gemm_multi), when the gradient is first needed: by the producer's own backward, by another writer, or
    # at a sync, a region's end or a graph cut. Same terms, added in the same order.
    def _deferDx(self, e: _Entry, rows: int, cols: int, dy: int, w: int, K: int):
        if e.pendingDx is None:
            e.pendingDx = (rows, cols, [])
            self._pendingDx[id(e)] = e
        e.pendingDx[2].append((dy, w, K))
        if len(e.pendingDx[2]) == 8 or not self.mergeInputGradients:
            self._flushDx(e)

    # `add` backward hands the upstream gradient to both inputs (src/model/autograd.ts:382-397): two copies of a
    # [T, hidden] buffer per residual connection. Here an input whose gradient has not been written yet only notes the
    # upstream address (`copyFrom`). Readers of that gradient read the upstream buffer in place, and the one writer
    # that follows in a transformer block, the norm's backward, adds its term on top of it while writing the real
    # buffer (gt_rmsnorm_bwd_add). Any other writer makes the copy, and so does every point where the upstream buffer
    # may be recycled while the entry lives on (a region's end, a reclaim). The gradient of an op's OUTPUT (the
    # projection on the other side of the residual connection) is only ever read by that op's backward, in place: where
    # gradients are handed to someone outside the ops (an optimizer, an exchange, a sync) only parameters matter, so the
    # copy into a transient's gradient is not made there (60 copies of [T, hidden] per step of a 30-layer model).
    def _materializeCopy(self, e: _Entry):
        self._check(self.lib.gt_copy(self.ctx, self._gradAddr(e), e.copyFrom, e.bytes))
        e.copyFrom = 0
        e.gradLive = True
        self._pendingCopy.pop(id(e), None)

    def _flushAllCopies(self, transients: str = "copy"):
        """`transients`: what to do with notes on gradients of op outputs: "copy" (make them), "keep" (leave them
        noted: nothing is being recycled) or "drop" (their entries are about to be recycled with the upstream buffers)."""
        for e in list(self._pendingCopy.values()):
            if e.external or transients == "copy":
                self._materializeCopy(e)
            elif transients == "drop":
                e.copyFrom = 0
                self._pendingCopy.pop(id(e), None)

    def _flushDx(self, e: _Entry):
        if e.copyFrom:
            self._materializeCopy(e)
        rows, cols, parts = e.pendingDx
        e.pendingDx = None
        self._pendingDx.pop(id(e), None)
        acc = 1 if e.gradLive else 0
        e.gradLive = True
        self._gradAddr(e)
        n = len(parts)
        if n == 1:
            self._gemm("NN", acc, rows, cols, parts[0][2], parts[0][0], parts[0][1], e.grad)
            return
        Ks = _I32[n](*[p[2] for p in parts])
        As = _U64[n](*[p[0] for p in parts])
        Bs = _U64[n](*[p[1] for p in parts])
        self._check(self.lib.gt_gemm_multi(self.ctx, _KIND["NN"], acc, rows, cols, n, Ks, As, Bs, e.grad))

    # Projections of the same activation (q, k and v of the normed input; gate and up) are noted when recorded and
    # launched together when the first of their outputs is needed: q/k/v as one grouped product (gt_gemm_grouped), gate and
    # up, when a gated unit consumes both, as one launch that also applies the unit (gt_glu_linear_fwd, see _gatedUnit).
    def _deferLinear(self, ex: _Entry, ew: _Entry, eo: _Entry, T: int, inDim: int, outDim: int):
        first = self._pendingFwd[0] if self._pendingFwd else None
        if first is not None and ("norm" in first or "lora" in first or first["ex"] is not ex or len(self._pendingFwd) == 8):
            self._flushFwd()
        self._pendingFwd.append({"ex": ex, "ew": ew, "eo": eo, "T": T, "inDim": inDim, "outDim": outDim})
        eo.pendingFwd = True

    # A per-head norm (q and k of the Qwen3 and Gemma 3 blocks) waits the same way for the rotary embedding that follows
    # it: if that is its first reader, one pass normalises and rotates (gt_rmsnorm_heads_rope_fwd).
    def _deferHeadNorm(self, ex: _Entry, ew: _Entry, eo: _Entry, rinv: int, T: int, H: int, hd: int, eps: float):
        first = self._pendingFwd[0] if self._pendingFwd else None
        if first is not None and ("norm" not in first or len(self._pendingFwd) == 8):
            self._flushFwd()
        self._pendingFwd.append(dict(norm=True, ex=ex, ew=ew, eo=eo, rinv=rinv, T=T, H=H, hd=hd, eps=eps, outDim=H * hd))
        eo.pendingFwd = True

    def _flushFwd(self):
        parts = self._pendingFwd
        if not parts:
            return
        self._pendingFwd = []
        for p in parts:
            p["eo"].pendingFwd = False
        if "lora" in parts[0]:
            n = len(parts)
            p0 = parts[0]
            T, inDim, r, s = p0["T"], p0["inDim"], p0["r"], p0["s"]
            if n == 1:
                self._check(self.lib.gt_gemm_scaled(self.ctx, _KIND["NT"], 0, T, r, inDim, p0["ex"].data, p0["ea"].data, p0["ts"], s))
            else:
                Ms, Ns = _I32[n](*([T] * n)), _I32[n](*([r] * n))
                As = _U64[n](*([p0["ex"].data] * n))
                Bs = _U64[n](*[p["ea"].data for p in parts])
                Cs = _U64[n](*[p["ts"] for p in parts])
                acc = _I32[n](*([0] * n))
                self._check(self.lib.gt_gemm_grouped_scaled(self.ctx, _KIND["NT"], n, Ms, Ns, inDim, As, Bs, Cs, acc, s))
            for p in parts:
                self._gemm2("NT", 0, T, p["outDim"], inDim, p["ex"].data, p["ew"].data, r, p["ts"], p["eb"].data, p["eo"].data)
            return
        if "norm" in parts[0]:
            for p in parts:
                T, H, hd = p["T"], p["H"], p["hd"]
                plain = (lambda p=p: self._check(self.lib.gt_rmsnorm_fwd(self.ctx, p["T"] * p["H"], p["hd"], p["ex"].data, p["ew"].data,
                                                                          p["eps"], p["eo"].data, p["rinv"])))
                if "rope" in p:
                    er, _H, _hd, base, posOffset = p["rope"]
                    er.pendingFwd = False
                    self._check(self.lib.gt_rmsnorm_heads_rope_fwd(self.ctx, T, H, hd, p["ex"].data, p["ew"].data, p["eps"], er.data,
                                                                   p["rinv"], float(base), posOffset))
                    p["eo"].lazy = plain        # (the same row statistics are written again if it ever runs)
                else:
                    plain()
            return
        n = len(parts)
        T, inDim = parts[0]["T"], parts[0]["inDim"]
        roped = [p for p in parts if "rope" in p]
        if roped:
            # projections whose one reader so far is a rotary embedding: the launch writes the rotated values into the
            # embedding's output; the projection's own buffer stays unwritten unless someone else asks for it
            _er, _H, hd, base, posOffset = roped[0]["rope"]
            for p in roped:
                p["rope"][0].pendingFwd = False
                p["eo"].lazy = (lambda p=p: self._gemm("NT", 0, p["T"], p["outDim"], p["inDim"], p["ex"].data, p["ew"].data, p["eo"].data))
            Ns = _I32[n](*[p["outDim"] for p in parts])
            Ws = _U64[n](*[p["ew"].data for p in parts])
            Ys = _U64[n](*[(p["rope"][0].data if "rope" in p else p["eo"].data) for p in parts])
            Hs = _I32[n](*[(p["rope"][1] if "rope" in p else 0) for p in parts])
            self._check(self.lib.gt_linear_rope_grouped(self.ctx, n, T, inDim, parts[0]["ex"].data, Ns, Ws, Ys, Hs, hd, float(base), posOffset))
            return
        if n == 1:
            self._gemm("NT", 0, T, parts[0]["outDim"], inDim, parts[0]["ex"].data, parts[0]["ew"].data, parts[0]["eo"].data)
            return
        Ms = _I32[n](*([T] * n))
        Ns = _I32[n](*[p["outDim"] for p in parts])
        As = _U64[n](*[p["ex"].data for p in parts])
        Bs = _U64[n](*[p["ew"].data for p in parts])
        Cs = _U64[n](*[p["eo"].data for p in parts])
        acc = _I32[n](*([0] * n))
        self._check(self.lib.gt_gemm_grouped(self.ctx, _KIND["NT"], n, Ms, Ns, inDim, As, Bs, Cs, acc))

    def _materializeLazy(self, e: _Entry):
        launch = e.lazy
        e.lazy = None
        launch()

    def _flushAllDx(self, transients: str = "copy"):
        self._flushFwd()
        for e in list(self._pendingDx.values()):
            self._flushDx(e)
        self._flushAllCopies(transients)
        self._flushDw()

    # The weight gradient of `linear` is dW (+)= dY^T.X: a small output (out x in) contracted over every row. Each has
    # too few output tiles to fill the GPU, so each is cut along K into slices, with a clear before, partial sums
    # combined in L2 and a last wave of its own. Up to eight of them (the projections of a layer) are launched together
    # as one grouped product (gt_gemm_grouped): their tiles share the SMs and one split-K factor. A closure notes its
    # (dY, X, dW); the group is launched when it is full, before anything else touches one of its gradients, and at
    # every point where buffers may be recycled or gradients are handed over (sync, region end, graph cut, optimizer).
    def _deferDw(self, ew: _Entry, gw: int, accum: int, rows: int, outDim: int, inDim: int, dy: int, x: int):
        if self._pendingDw and (self._pendingDwRows != rows or len(self._pendingDw) == 8):
            self._flushDw()
        self._pendingDwRows = rows
        self._pendingDw.append((dy, x, gw, accum, outDim, inDim, ew))
        ew.pendingDw = True

    def _flushDw(self):
        parts = self._pendingDw
        if not parts:
            return
        self._pendingDw = []
        rows = self._pendingDwRows
        for p in parts:
            p[6].pendingDw = False
        n = len(parts)
        if n == 1:
            dy, x, gw, acc, outDim, inDim, _e = parts[0]
            self._gemm("TN", acc, outDim, inDim, rows, dy, x, gw)
            return
        Ms = _I32[n](*[p[4] for p in parts])
        Ns = _I32[n](*[p[5] for p in parts])
        As = _U64[n](*[p[0] for p in parts])
        Bs = _U64[n](*[p[1] for p in parts])
        Cs = _U64[n](*[p[2] for p in parts])
        acc = _I32[n](*[p[3] for p in parts])
        self._check(self.lib.gt_gemm_grouped(self.ctx, _KIND["TN"], n, Ms, Ns, rows, As, Bs, Cs, acc))

    def flushDeferred(self):
        """Launch everything whose launch was put off (merged input gradients, grouped weight gradients, copies):
        called by whoever is about to use gradients outside the ops, e.g. an optimizer step or a gradient exchange."""
        self._flushAllDx("keep")

    def _gradTarget(self, t: Tensor, e: _Entry):
        """(grad address or 0, accum flag) for a backward kernel about to write into t's gradient."""
        if not self._flows(t, e):
            return 0, 0
        if e.pendingDw:
            self._flushDw()             # an earlier product into this gradient goes first
        if e.copyFrom:
            self._materializeCopy(e)
        if e.pendingDx is not None:
            self._flushDx(e)
        acc = 1 if e.gradLive else 0
        e.gradLive = True
        return e.grad or self._gradAddr(e), acc

    def _gradSource(self, e: _Entry) -> int:
        """The upstream gradient of an op output. Never written means it is exactly zero."""
        if e.pendingDw:
            self._flushDw()
        if e.pendingDx is not None:
            self._flushDx(e)           # (a gradient that is still a view gets its copy made first: _flushDx writes into it)
        if e.copyFrom:
            return e.copyFrom          # still exactly the upstream buffer of an `add`: read it there, no copy
        if not e.gradLive:
            self._check(self.lib.gt_zero(self.ctx, self._gradAddr(e), e.bytes))
            self.gradClearsIssued += 1
            e.gradLive = True
        return e.grad

    # ------------------------------------------------------------------ data movement
    def uploadParams(self, tensors: Sequence[Tensor]):
        """webgpu.ts:406-411."""
        for t in tensors:
            e = self._entryFor(t)
            self._write(e.data, t.data)

    def reserveGradArena(self, tensors: Sequence[Tensor]) -> tuple:
        """Give the listed trainable tensors gradient buffers carved, in order, from one contiguous
        block, so a data-parallel step can sum them across ranks in a few large buckets.
        Returns (address, element count, [offset per tensor])."""
        total = 0
        offs = []
        for t in tensors:
            if self._find(t) is not None:
                raise _lib.GtError(4, "reserveGradArena must run before the tensors are first used")
            offs.append(total)
            total += (t.size + 63) // 64 * 64   # 256-byte aligned slices
        base = self.createStateBuffer(total * 4)
        for t, off in zip(tensors, offs):
            e = self._newExternal(t, self._acquirePersistent(t.size * 4), base + off * 4)
            self._write(e.data, t.data)
        return base, total, offs

    def sync(self, reads: Sequence[Tensor] = ()):
        """webgpu.ts:419-576: flush, copy back `reads` and the gradients of every touched external that
        requires grad and is not kept on device, recycle the transients."""
        if self._capturing:
            raise _lib.GtError(4, "sync() inside a graph capture")
        self._readback = 0
        self._flushAllDx("drop")
        self._flushPendingActs(only=list(reads))
        self._pendingAct.clear()
        self._pendingAdd.clear()
        seen = set()
        wanted = []                            # (address, host array)
        for t in reads:
            if id(t) in seen:
                continue
            seen.add(id(t))
            e = self._find(t)
            if e is None:
                continue
            if e.lazy is not None:
                self._materializeLazy(e)
            wanted.append((e.data, t.dataForReading()))
        for t in self._touched:
            e = self._find(t)
            if e is None:
                continue
            e.touched = False
            if t.requiresGrad and e.grad:
                if not e.gradLive:
                    # touched by a forward, never written by a backward: the reference's cleared buffer
                    self._check(self.lib.gt_zero(self.ctx, e.grad, e.bytes))
                    self.gradClearsIssued += 1
                if t not in self._keptOnDevice:
                    wanted.append((e.grad, t.gradForReading()))
            if e.gradLive:
                e.gradLive = False   # the next graph's first writer overwrites (the deferred clear)
        self._readMany(wanted)
        self._check(self.lib.gt_sync(self.ctx))
        self.lastSyncReadbackBytes = self._readback
        for blocks in (self._transients, self._regionFree, self._outer):
            for addr, size in blocks:
                self._release(addr, size)
        self._transients, self._regionFree, self._outer = [], [], []
        self._dropTape()
        self._regionStack = []
        self._touched = []
        self._backwardBegun = False
        if self._graphOpen:                    # (a sync with no graph behind it, e.g. after building an optimizer, arms nothing)
            self._graphSynced = True
        self._graphOpen = False
        self._regionRecs.clear()
        self._curRec = None
        self._regionDepth = 0

    def reclaimStepTransients(self, keep: Sequence[Tensor] = ()):
        """webgpu.ts:612-633: recycle this micro-batch's transients without the readback."""
        self._flushAllDx("drop")
        keepBufs = set()
        for t in keep:
            e = self._find(t)
            if e is not None:
                keepBufs.add(e.data)
        retained = []
        for tr in self._transients:
            if tr[0] in keepBufs:
                retained.append(tr)
            else:
                self._release(*tr)
        self._transients = retained
        for blocks in (self._regionFree, self._outer):
            for addr, size in blocks:
                self._release(addr, size)
        self._regionFree, self._outer = [], []
        self._dropTape()

    # ------------------------------------------------------------------ regions (RegionBackend)
    def beginRegion(self) -> int:
        self._regionsOpened += 1
        self._regionDepth += 1
        self._regionStack.append((self._regionsOpened, len(self._tape)))
        if self._regionDepth == 1 and self.keepAttentionAcrossRecompute:
            self._curRec = {"id": self._nextRegionId, "saved": [], "pos": 0, "replay": False}
            self._nextRegionId += 1
        else:
            if self._curRec is not None:             # a region inside a region: nothing is kept for either
                self._regionRecs.pop(self._curRec["id"], None)
            self._curRec = None
        return len(self._transients)

    # Optional extension of RegionBackend, used by `checkpoint` when present. A recompute region runs its forward
    # twice; the attention inside it is the one op whose second run costs real time (a quarter of a layer's forward)
    # while its result is, by construction, bit-identical to the first. So the first run's attention outputs (O and
    # the row statistics) survive the region's end, and the replay, told which region it repeats, takes them instead
    # of launching the kernel again. Everything else of the region is still freed and recomputed.
    def regionToken(self) -> Optional[int]:
        """Identity of the outermost region just opened (None when nothing will be kept for it)."""
        rec = self._curRec
        if rec is None or rec["replay"]:
            return None
        self._regionRecs[rec["id"]] = rec
        return rec["id"]

    def replayOf(self, token: Optional[int]):
        """The region just opened repeats the forward of region `token`."""
        rec = self._regionRecs.get(token) if token is not None else None
        if rec is not None and self._regionDepth == 1:
            rec["replay"], rec["pos"] = True, 0
            self._curRec = rec

    def regionCount(self) -> int:
        return self._regionsOpened

    def endRegion(self, mark: int, keep: Sequence[Tensor]):
        """webgpu.ts:659-702."""
        if mark > len(self._transients):
            raise RuntimeError(
                f"endRegion: mark {mark} is past the {len(self._transients)} live transients; "
                f"a sync() or reclaim ran inside the region")
        self._flushAllDx()
        self._flushPendingActs(only=list(keep))
        _serial, tapeMark = self._regionStack.pop() if self._regionStack else (0, len(self._tape))
        outer = self._regionStack[-1][0] if self._regionStack else 0
        self._dropTape(tapeMark, keep)
        keepBufs = set()
        for t in keep:
            e = self._find(t)
            if e is not None:
                keepBufs.add(e.data)
                keepBufs.add(e.grad)
                e.region = outer
                self._tape.append(t)
        rec = self._curRec if self._regionDepth == 1 else None
        self._regionDepth = max(0, self._regionDepth - 1)
        release = set()
        if rec is not None:
            self._curRec = None
            held = {b for item in rec["saved"] for b in item[:2]}
            if rec["replay"]:
                release = held                       # the replay and its backward are over: the kept outputs go too
                self._regionRecs.pop(rec["id"], None)
            elif rec["id"] in self._regionRecs:
                keepBufs |= held                     # first run, and `checkpoint` asked for a token: keep them
        retained = []
        for tr in self._transients[:mark]:
            if tr[0] in release:
                self._regionFree.append(tr)
            else:
                retained.append(tr)
        for tr in self._transients[mark:]:
            if tr[0] in keepBufs:
                retained.append(tr)
            else:
                self._regionFree.append(tr)
        self._transients = retained

    def seedGradFrom(self, dst: Tensor, src: Tensor):
        """webgpu.ts:748-761."""
        self._ensureBackwardBegun()
        ed, es = self._entryOf(dst), self._entryOf(src)
        if ed is None or es is None:
            raise RuntimeError("seedGradFrom: tensor has no GPU buffers")
        if dst.size != src.size:
            raise RuntimeError(f"seedGradFrom: size mismatch {dst.size} vs {src.size}")
        self._check(self.lib.gt_copy(self.ctx, self._gradAddr(ed), self._gradSource(es), src.size * 4))
        ed.gradLive = True

    def seedGradFromHost(self, t: Tensor):
        """webgpu.ts:1432-1437."""
        self._ensureBackwardBegun()
        e = self._entryOf(t)
        if e is None:
            raise RuntimeError("seedGradFromHost: tensor has no GPU buffers")
        self._write(self._gradAddr(e), t.grad)
        e.gradLive = True

    def _beginForwardOp(self, keepPending: bool = False):
        """Every forward op starts here. Unless the op launches nothing itself (`keepPending`), projections noted but
        not launched yet go first, so no kernel can read an output that does not exist yet."""
        if self._pendingFwd and not keepPending:
            self._flushFwd()
        self._backwardBegun = False
        self._graphSynced = False
        self._graphOpen = True

    def _ensureBackwardBegun(self):
        """webgpu.ts:1397-1429. A sync() between a graph's forward and its backward recycled the graph's
        buffers; refuse to accumulate into them."""
        if self._pendingFwd:
            self._flushFwd()
        if self._backwardBegun:
            return
        if self._graphSynced:
            raise RuntimeError(
                "backward over a graph built before a sync(): that sync recycled the graph's "
                "gradient buffers and discarded their clears, so this backward would "
                "accumulate into pool garbage")
        self._backwardBegun = True

    # ------------------------------------------------------------------ raw buffers (optimizers, checkpoints)
    def buffersFor(self, t: Tensor):
        e = self._entryFor(t)
        if e.copyFrom:                  # the caller is about to look at the gradient buffer itself
            self._materializeCopy(e)
        return {"data": e.data, "grad": e.grad}

    def keepGradOnDevice(self, t: Tensor):
        self._keptOnDevice.add(t)

    def createStateBuffer(self, nbytes: int) -> int:
        out = C.c_uint64()
        self._check(self.lib.gt_alloc_state(self.ctx, nbytes, C.byref(out)))
        self._stateBufs[int(out.value)] = nbytes
        return int(out.value)

    def writeStateBuffer(self, buf: int, f32: np.ndarray):
        self._write(buf, np.ascontiguousarray(f32, dtype=np.float32))

    def readStateBuffer(self, buf: int, n: int) -> np.ndarray:
        out = np.empty(n, np.float32)
        self._read(buf, out)
        return out

    # ------------------------------------------------------------------ asynchronous reads (checkpoints)
    def readAsync(self, addr: int, nbytes: int) -> int:
        """Start copying `nbytes` at `addr`, as of the work enqueued so far, to pinned host memory on a copy stream
        that runs beside later compute. Returns a ticket for `readFinish`."""
        t = C.c_uint64()
        self._check(self.lib.gt_read_async(self.ctx, addr, nbytes, C.byref(t)))
        return int(t.value)

    def readFence(self):
        """Later compute waits (on the device) for every read started so far: call before work that overwrites their
        sources. The optimizers call it at the top of `recordStep`."""
        self._check(self.lib.gt_read_fence(self.ctx))

    def readFinish(self, ticket: int, out: np.ndarray):
        assert out.flags["C_CONTIGUOUS"]
        self._check(self.lib.gt_read_finish(self.ctx, ticket, out.ctypes.data, out.nbytes))

    # ------------------------------------------------------------------ graph capture
    def beginCapture(self, seed: float = 1.0, accumulate: bool = True):
        """Start recording device work into a replayable graph. Run the same work once eagerly first:
        recording cannot allocate (the pool, RoPE tables and scratch must already be warm).
        `seed` is the loss seed the recorded backward uses. With `accumulate` the recorded backward adds
        into the parameter gradients (replay it once per micro-batch after zeroing them); without, its
        first write to each parameter gradient overwrites (one replay per step)."""
        if self._capturing:
            raise _lib.GtError(4, "beginCapture: already capturing")
        if self._seedBuf == 0:
            self._seedBuf = self.createStateBuffer(4)
        self._write(self._seedBuf, np.array([seed], np.float32))
        for e in self._externals.values():
            if e.grad:
                e.gradLive = bool(accumulate)
        self._check(self.lib.gt_graph_begin(self.ctx))
        self._capturing = True
        self._captureInputs = []
        self._captureSegments = []
        self._captureMark = len(self._transients)
        self._outerMark = len(self._outer)

    def cutCapture(self) -> int:
        """Close the graph recorded so far and start the next one: the place where the replayer will issue work from
        the host between two segments. Returns the number of segments closed so far."""
        if not self._capturing:
            raise _lib.GtError(4, "cutCapture: not capturing")
        self._flushAllDx("keep")
        h = C.c_uint64()
        self._check(self.lib.gt_graph_end(self.ctx, C.byref(h)))
        self._captureSegments.append(int(h.value))
        self._check(self.lib.gt_graph_begin(self.ctx))
        return len(self._captureSegments)

    def endCapture(self, outputs: Optional[Dict[str, Tensor]] = None) -> CapturedGraph:
        h = C.c_uint64()
        self._flushAllDx("drop")
        self._capturing = False
        self._check(self.lib.gt_graph_end(self.ctx, C.byref(h)))
        owned = self._transients[self._captureMark:] + self._regionFree + self._outer[self._outerMark:]
        self._transients = self._transients[:self._captureMark]
        self._outer = self._outer[:self._outerMark]
        self._regionFree = []
        self._dropTape()
        owned = owned + [(a, max(256, (n * 4 + 255) & ~255)) for a, n, _r, _b in self._captureInputs]
        outs = {}
        for name, t in (outputs or {}).items():
            e = self._entries[t]
            outs[name] = (e.data, t.size)
        g = CapturedGraph(self, int(h.value), list(self._captureInputs), owned, outs, earlier=self._captureSegments)
        self._captureInputs = []
        self._captureSegments = []
        # externals touched while recording keep their accumulate-or-overwrite state as recorded
        return g

    def readGraphOutput(self, g: CapturedGraph, name: str) -> np.ndarray:
        addr, n = g.outputs[name]
        out = np.empty(n, np.float32)
        self._read(addr, out)
        return out

    # ------------------------------------------------------------------ events
    def recordEvent(self, slot: int):
        self._check(self.lib.gt_event_record(self.ctx, slot))

    def elapsedMs(self, a: int, b: int) -> float:
        ms = C.c_float()
        self._check(self.lib.gt_event_elapsed_ms(self.ctx, a, b, C.byref(ms)))
        return float(ms.value)

    # ------------------------------------------------------------------ ops (OpsBackend)
    def _gemm(self, kind: str, accum: int, M: int, N: int, K: int, a: int, b: int, c: int):
        self._check(self.lib.gt_gemm(self.ctx, _KIND[kind], accum, M, N, K, a, b, c))

    def _gemm2(self, kind: str, accum: int, M: int, N: int, K: int, a: int, b: int, K2: int, a2: int, b2: int, c: int):
        self._check(self.lib.gt_gemm2(self.ctx, _KIND[kind], accum, M, N, K, a, b, K2, a2, b2, c))

    def linear(self, x: Tensor, w: Tensor) -> Tensor:
        """webgpu.ts:884-903."""
        self._beginForwardOp(keepPending=True)
        T, inDim = x.shape
        outDim = w.shape[0]
        ex, ew = self._entryFor(x), self._entryFor(w)
        needs = self._flows(x, ex) or self._flows(w, ew)
        out, eo = self._makeOut([T, outDim], T * outDim, [x, w], needs)
        if self.groupForward:
            self._deferLinear(ex, ew, eo, T, inDim, outDim)
        else:
            self._flushFwd()
            self._gemm("NT", 0, T, outDim, inDim, ex.data, ew.data, eo.data)
        return self._record(out, needs, self._linearBackward, x, ex, w, ew, eo, T, inDim, outDim)

    def _linearBackward(self, x, ex, w, ew, eo, T, inDim, outDim):
        self._ensureBackwardBegun()
        go = self._gradSource(eo)
        if self._flows(x, ex):
            self._deferDx(ex, T, inDim, go, ew.data, outDim)
        if self._flows(w, ew):
            gw, aw = self._gradTarget(w, ew)
            # (a product with many output tiles, the readout's, fills the GPU alone and is launched as it comes)
            if self.groupWeightGradients and ((outDim + 255) // 256) * ((inDim + 191) // 192) <= 64:
                self._deferDw(ew, gw, aw, T, outDim, inDim, go, ex.data)
            else:
                self._gemm("TN", aw, outDim, inDim, T, go, ex.data, gw)

    def loraLinear(self, x: Tensor, w: Tensor, a: Tensor, b: Tensor, scale: float) -> Tensor:
        """The adapter-carrying projection of autograd.ts:311-319, y = x·Wᵀ + scale·((x·Aᵀ)·Bᵀ), as one op. Recorded as
        `add(linear(x,w), scale(linear(linear(x,a),b), scale))` it costs two more passes over [T, out] in forward
        (scale, add) and two in backward; here the factor is applied to the [T, r] intermediate instead and the
        low-rank product is r more columns of the wide product's contraction (`gt_gemm2`), so [T, out] is written
        once and not read back. (scale·t)·Bᵀ equals scale·(t·Bᵀ) up to rounding, exactly when scale is a power of two, e.g. the
        usual alpha/r = 2.) Gradients: dx += g·W + (scale·(g·B))·A, dB += gᵀ·(scale·t), dA += (scale·(g·B))ᵀ·x,
        and dW += gᵀ·x when the base weight is not frozen."""
        self._beginForwardOp(keepPending=self.groupForward)
        T, inDim = x.shape
        outDim, r = w.shape[0], a.shape[0]
        ex, ew, ea, eb = self._entryFor(x), self._entryFor(w), self._entryFor(a), self._entryFor(b)
        needs = self._flows(x, ex) or self._flows(w, ew) or self._flows(a, ea) or self._flows(b, eb)
        out, eo = self._makeOut([T, outDim], T * outDim, [x, w, a, b], needs)
        small = T * r * 4
        ts, dt = self._acquireRecycled(small), self._acquireRecycled(small)
        s = float(scale)
        kNT, kNN = _KIND["NT"], _KIND["NN"]
        if self.groupForward:
            # noted, not launched: projections of the same input (q, k, v; gate, up) form their thin products
            # ts = scale·(x·Aᵀ) in one grouped launch, which reads x once (_flushFwd)
            first = self._pendingFwd[0] if self._pendingFwd else None
            if first is not None and ("lora" not in first or first["ex"] is not ex or first["r"] != r or first["s"] != s
                                      or len(self._pendingFwd) == 8):
                self._flushFwd()
            self._pendingFwd.append(dict(lora=True, ex=ex, ew=ew, ea=ea, eb=eb, eo=eo, ts=ts, T=T, inDim=inDim, outDim=outDim, r=r, s=s))
            eo.pendingFwd = True
        else:
            # ts = scale·(x·Aᵀ): the factor rides on the product's epilogue (gt_gemm_scaled), no pass of its own
            self._check(self.lib.gt_gemm_scaled(self.ctx, kNT, 0, T, r, inDim, ex.data, ea.data, ts, s))
            self._gemm2("NT", 0, T, outDim, inDim, ex.data, ew.data, r, ts, eb.data, eo.data)

        def _bw():
            self._ensureBackwardBegun()
            go = self._gradSource(eo)
            wantDx = self._flows(x, ex)
            self._check(self.lib.gt_gemm_scaled(self.ctx, kNN, 0, T, r, outDim, go, eb.data, dt, s))   # dt = scale·(g·B)
            # dB = gᵀ·ts and dA = dtᵀ·x: thin outputs contracted over every row, bound by reading g and x; the fourteen of a
            # layer go out as two grouped launches (_deferDw) instead of one launch each
            if b.requiresGrad:
                gb, ab = self._gradTarget(b, eb)
                if gb:
                    if self.groupWeightGradients:
                        self._deferDw(eb, gb, ab, T, outDim, r, go, ts)
                    else:
                        self._gemm("TN", ab, outDim, r, T, go, ts, gb)
            if a.requiresGrad:
                ga, aa = self._gradTarget(a, ea)
                if ga:
                    if self.groupWeightGradients:
                        self._deferDw(ea, ga, aa, T, r, inDim, dt, ex.data)
                    else:
                        self._gemm("TN", aa, r, inDim, T, dt, ex.data, ga)
            if wantDx:      # g·W + dt·A: two more K ranges of x's input-gradient product
                self._deferDx(ex, T, inDim, go, ew.data, outDim)
                self._deferDx(ex, T, inDim, dt, ea.data, r)
            if w.requiresGrad:
                gw, aw = self._gradTarget(w, ew)
                if gw:
                    self._gemm("TN", aw, outDim, inDim, T, go, ex.data, gw)

        return self._record(out, needs, _bw)

    def _elementwise(self, op: str, a: Tensor, b: Optional[Tensor], c: float) -> Tensor:
        self._beginForwardOp()
        ea = self._entryFor(a)
        eb = self._entryFor(b) if b is not None else None
        needs = self._flows(a, ea) or (eb is not None and self._flows(b, eb))
        out, eo = self._makeOut(list(a.shape), a.size, [a, b] if b is not None else [a], needs)
        n = a.size
        code = _EW[op]
        self._check(self.lib.gt_ew_fwd(self.ctx, code, n, ea.data, eb.data if eb else 0, c, eo.data))

        def _bw():
            self._ensureBackwardBegun()
            go = self._gradSource(eo)
            if eb is not None and eb is ea:
                # add(t,t) / mul(t,t): both contributions land in one buffer, summed in one write
                ga, aa = self._gradTarget(a, ea)
                self._check(self.lib.gt_ew_bwd(self.ctx, code, n, ea.data, ea.data, c, go, ga, aa, ga, aa))
                return
            ga, aa = self._gradTarget(a, ea)
            gb, ab = self._gradTarget(b, eb) if eb is not None else (0, 0)
            self._check(self.lib.gt_ew_bwd(self.ctx, code, n, ea.data, eb.data if eb else 0, c, go, ga, aa, gb, ab))

        return self._record(out, needs, _bw)

    def add(self, a, b):
        """webgpu.ts:905-960. Not launched when recorded: if the first use of the sum is a norm (every residual
        connection of a block), one kernel forms the sum and normalises it (gt_add_rmsnorm_fwd); any other use
        launches the plain add then. Backward launches nothing where it can (see _materializeCopy)."""
        if a is b or not self.fuseResidualNorm or a.shape != b.shape:
            return self._elementwise("add", a, b, 0.0)
        self._beginForwardOp(keepPending=True)
        ea, eb = self._entryFor(a), self._entryFor(b)
        out = Tensor.output(list(a.shape), a.size, [a, b])
        out._needs = self._flows(a, ea) or self._flows(b, eb)
        self._pendingAdd[id(out)] = (out, a, b)
        return self._record(out, out._needs, self._addBackward, out, a, ea, b, eb)

    def _addBackward(self, out, a, ea, b, eb):
        eo = self._find(out)
        if eo is None:
            return          # never used by anything: no gradient reaches it
        self._ensureBackwardBegun()
        go = self._gradSource(eo)
        for t, e, first in ((a, ea, True), (b, eb, False)):
            if not self._flows(t, e):
                continue
            if e.pendingDx is not None:
                self._flushDx(e)
            if e.gradLive or e.copyFrom:
                g, acc = self._gradTarget(t, e)
                self._check(self.lib.gt_ew_bwd(self.ctx, _EW["add"], a.size, ea.data, eb.data, 0.0, go,
                                               g if first else 0, acc, 0 if first else g, acc))
            else:
                e.copyFrom = go
                self._pendingCopy[id(e)] = e

    def _materializeAdd(self, t: Tensor) -> _Entry:
        _t, a, b = self._pendingAdd.pop(id(t))
        ea, eb = self._find(a), self._find(b)
        self._flushFwd()
        e = self._newEntry(t, t._needs)
        self._check(self.lib.gt_ew_fwd(self.ctx, _EW["add"], t.size, ea.data, eb.data, 0.0, e.data))
        return e

    def mul(self, a, b):
        if a is not b:
            for act, other in ((a, b), (b, a)):
                if id(act) in self._pendingAct and id(other) not in self._pendingAct:
                    return self._gatedUnit(act, other)
        return self._elementwise("mul", a, b, 0.0)

    def silu(self, x):
        return self._activation("silu", x)

    def gelu(self, x):
        return self._activation("gelu", x)

    # An activation is not launched when it is recorded: if its only use turns out to be a product (the gated FFN
    # unit silu(gate)*up / gelu(gate)*up), one fused kernel does both and the activated gate is never written. Any
    # other use (another op, a sync that reads it, the end of a recompute region) launches it then, unchanged.
    def _activation(self, op: str, x: Tensor) -> Tensor:
        if not self.fuseGatedUnits:
            return self._elementwise(op, x, None, 0.0)
        self._beginForwardOp(keepPending=True)
        e0 = self._find(x)
        if e0 is None or not e0.pendingFwd:      # (a projection still waiting to be launched stays waiting: see _gatedUnit)
            e0 = self._entryFor(x)
        t = Tensor.output(list(x.shape), x.size, [x])
        t._needs = self._flows(x, e0)
        self._pendingAct[id(t)] = (t, _EW[op], x)
        return self._record(t, t._needs, self._activationBackward, t, op, x)

    def _activationBackward(self, t, op, x):
        e = self._find(t)
        if e is None or not (e.gradLive or e.copyFrom or e.pendingDx is not None):
            return          # consumed only by fused products, which sent their gradient straight to x
        self._ensureBackwardBegun()
        ex = self._entryOf(x)
        go = self._gradSource(e)
        gx, ax = self._gradTarget(x, ex)
        self._check(self.lib.gt_ew_bwd(self.ctx, _EW[op], x.size, ex.data, 0, 0.0, go, gx, ax, 0, 0))

    def _materializeAct(self, t: Tensor) -> _Entry:
        _t, code, x = self._pendingAct.pop(id(t))
        ex = self._find(x)
        self._flushFwd()
        if ex.lazy is not None:
            self._materializeLazy(ex)
        e = self._newEntry(t, t._needs)
        self._check(self.lib.gt_ew_fwd(self.ctx, code, t.size, ex.data, 0, 0.0, e.data))
        return e

    def _flushPendingActs(self, only=None):
        for key in list(self._pendingAct.keys()):
            t = self._pendingAct[key][0]
            if only is None or any(t is o for o in only):
                self._materializeAct(t)
        for key in list(self._pendingAdd.keys()):
            t = self._pendingAdd[key][0]
            if only is None or any(t is o for o in only):
                self._materializeAdd(t)

    def _gatedUnit(self, act: Tensor, u: Tensor) -> Tensor:
        _t, code, x = self._pendingAct[id(act)]
        self._beginForwardOp(keepPending=True)
        ex, eu = self._find(x), self._find(u)
        pend = self._pendingFwd
        if (eu is not None and len(pend) == 2 and ex.pendingFwd and eu.pendingFwd and ex is not eu
                and {id(pend[0]["eo"]), id(pend[1]["eo"])} == {id(ex), id(eu)} and pend[0]["outDim"] == pend[1]["outDim"]
                and "rope" not in pend[0] and "rope" not in pend[1] and "lora" not in pend[0]):
            # gate and up are the two projections waiting to be launched: one launch writes both and the gated unit
            pg, pu = (pend[0], pend[1]) if pend[0]["eo"] is ex else (pend[1], pend[0])
            self._pendingFwd = []
            ex.pendingFwd = eu.pendingFwd = False
            needs = self._flows(x, ex) or self._flows(u, eu)
            out, eo = self._makeOut(list(act.shape), act.size, [act, u], needs)
            self._check(self.lib.gt_glu_linear_fwd(self.ctx, code, pg["T"], pg["outDim"], pg["inDim"], pg["ex"].data, pg["ew"].data,
                                                   pu["ew"].data, ex.data, eu.data, eo.data))
        else:
            self._flushFwd()
            if ex.lazy is not None:
                self._materializeLazy(ex)
            eu = self._entryFor(u)
            needs = self._flows(x, ex) or self._flows(u, eu)
            out, eo = self._makeOut(list(act.shape), act.size, [act, u], needs)
            self._check(self.lib.gt_glu_fwd(self.ctx, code, act.size, ex.data, eu.data, eo.data))
        return self._record(out, needs, self._gatedUnitBackward, code, act.size, x, ex, u, eu, eo)

    def _gatedUnitBackward(self, code, n, x, ex, u, eu, eo):
        self._ensureBackwardBegun()
        go = self._gradSource(eo)
        gx, ax = self._gradTarget(x, ex)
        gu, au = self._gradTarget(u, eu)
        if gx and gx == gu:      # act(x) * x: one buffer takes both terms, in two passes
            self._check(self.lib.gt_glu_bwd(self.ctx, code, n, ex.data, eu.data, go, gx, ax, 0, 0))
            self._check(self.lib.gt_glu_bwd(self.ctx, code, n, ex.data, eu.data, go, 0, 0, gu, 1))
        else:
            self._check(self.lib.gt_glu_bwd(self.ctx, code, n, ex.data, eu.data, go, gx, ax, gu, au))

    def scale(self, x, c):
        return self._elementwise("scale", x, None, float(c))

    def _rmsNormRows(self, x: Tensor, w: Tensor, rows: int, d: int, eps: float, shape, heads=None) -> Tensor:
        """webgpu.ts:1673-1701. `heads` = (T, H): a per-head norm that may wait for the rotary embedding after it."""
        self._beginForwardOp(keepPending=heads is not None)
        ew = self._entryFor(w)
        if id(x) in self._pendingAdd and self._find(x) is None:
            # x = a + b has not been launched and this norm is its first use: one kernel writes both
            _t, a, b = self._pendingAdd.pop(id(x))
            ea, eb = self._find(a), self._find(b)
            ex = self._newEntry(x, x._needs)
            needs = self._flows(x, ex) or self._flows(w, ew)
            out, eo = self._makeOut(shape, x.size, [x, w], needs)
            rinv = self._acquireRecycled(rows * 4)
            self._check(self.lib.gt_add_rmsnorm_fwd(self.ctx, rows, d, ea.data, eb.data, ew.data, eps, ex.data, eo.data, rinv))
        else:
            ex = self._entryFor(x)
            needs = self._flows(x, ex) or self._flows(w, ew)
            out, eo = self._makeOut(shape, x.size, [x, w], needs)
            rinv = self._acquireRecycled(rows * 4)
            if heads is not None:
                self._deferHeadNorm(ex, ew, eo, rinv, heads[0], heads[1], d, eps)
            else:
                self._check(self.lib.gt_rmsnorm_fwd(self.ctx, rows, d, ex.data, ew.data, eps, eo.data, rinv))

        return self._record(out, needs, self._rmsNormBackward, x, ex, w, ew, eo, rinv, rows, d)

    def _rmsNormBackward(self, x, ex, w, ew, eo, rinv, rows, d):
        self._ensureBackwardBegun()
        go = self._gradSource(eo)
        wantX = self._flows(x, ex)
        if wantX and ex.pendingDx is not None:
            self._flushDx(ex)
        gw, aw = self._gradTarget(w, ew)
        if wantX and ex.copyFrom and not ex.gradLive:
            # the gradient so far is an `add`'s upstream buffer: dx = that buffer + this term, written in one pass
            gadd = ex.copyFrom
            ex.copyFrom = 0
            self._pendingCopy.pop(id(ex), None)
            ex.gradLive = True
            self._check(self.lib.gt_rmsnorm_bwd_add(self.ctx, rows, d, ex.data, ew.data, rinv, go, gadd, self._gradAddr(ex), gw, aw))
            return
        gx, ax = self._gradTarget(x, ex)
        self._check(self.lib.gt_rmsnorm_bwd(self.ctx, rows, d, ex.data, ew.data, rinv, go, gx, ax, gw, aw))

    def rmsNorm(self, x, weight, eps):
        T, d = x.shape
        return self._rmsNormRows(x, weight, T, d, eps, [T, d])

    def rmsNormHeads(self, x, weight, T, H, hd, eps):
        wait = self.fuseRope and hd in (64, 128, 256) and not (id(x) in self._pendingAdd and self._find(x) is None)
        return self._rmsNormRows(x, weight, T * H, hd, eps, [T, H * hd], heads=(T, H) if wait else None)

    def embedding(self, weight: Tensor, ids) -> Tensor:
        """webgpu.ts:1090-1108."""
        self._beginForwardOp()
        d = weight.shape[1]
        T = len(ids)
        ew = self._entryFor(weight)
        idBuf = self._uploadU32(ids, "ids", weight.shape[0])
        needs = self._flows(weight, ew)
        out, eo = self._makeOut([T, d], T * d, [weight], needs)
        self._check(self.lib.gt_embedding_fwd(self.ctx, T, d, ew.data, idBuf, eo.data))

        def _bw():
            self._ensureBackwardBegun()
            if not weight.requiresGrad or not ew.grad:
                return
            go = self._gradSource(eo)
            if ew.pendingDw:
                self._flushDw()
            if ew.pendingDx is not None:
                self._flushDx(ew)
            if ew.copyFrom:
                self._materializeCopy(ew)
            if not ew.gradLive:
                self._check(self.lib.gt_zero(self.ctx, ew.grad, ew.bytes))
                self.gradClearsIssued += 1
                ew.gradLive = True
            self._check(self.lib.gt_embedding_bwd(self.ctx, T, d, go, idBuf, ew.grad))

        return self._record(out, needs, _bw)

    def _checkT(self, T: int, rows: int, where: str):
        b, sl = self._batch
        if b and T != b * sl:
            raise ValueError(f"{where}: T={T} but the batch is {b} x {sl}")
        if not b and T != rows:
            raise ValueError(f"{where}: T={T} but the tensor has {rows} rows")

    def rope(self, x: Tensor, T: int, H: int, hd: int, base: float, posOffset: int = 0) -> Tensor:
        """webgpu.ts:1110-1123. Where the input is a projection that has not been launched yet (`rope(linear(x, Wq))`, the
        llama block) and the heads are 64 wide, the rotation is applied by the projection's launch as its tiles are
        written (gt_linear_rope_grouped); where it is a per-head norm that has not been launched yet (the Qwen3 and
        Gemma 3 blocks), by the norm's pass (gt_rmsnorm_heads_rope_fwd). No pass of its own runs in either case; the
        gradient side is in `attention`."""
        self._checkT(T, x.shape[0], "rope")
        e0 = self._find(x)
        part = None
        if self.fuseRope and e0 is not None and e0.pendingFwd:
            part = next((p for p in self._pendingFwd if p["eo"] is e0), None)
            if part is not None and "norm" in part:
                # a per-head norm waiting to be launched: it normalises and rotates in one pass
                if "rope" in part or (part["T"], part["H"], part["hd"]) != (T, H, hd):
                    part = None
            elif part is not None:
                # a projection waiting to be launched (64-wide heads, tensor-core mode): its launch writes the rotated values
                first = next((p["rope"] for p in self._pendingFwd if "rope" in p), None)
                if ("rope" in part or "lora" in part or part["outDim"] != H * hd or hd != 64 or self.precision != "tf32" or T < 16 or
                        (first is not None and first[2:] != (hd, base, posOffset))):
                    part = None
        if part is not None:
            self._beginForwardOp(keepPending=True)
            ex = e0
            needs = self._flows(x, ex)
            out, eo = self._makeOut([T, H * hd], T * H * hd, [x], needs)
            part["rope"] = (eo, H, hd, base, posOffset)
            eo.pendingFwd = True
        else:
            self._beginForwardOp()
            ex = self._entryFor(x)
            needs = self._flows(x, ex)
            out, eo = self._makeOut([T, H * hd], T * H * hd, [x], needs)
            self._check(self.lib.gt_rope_fwd(self.ctx, T, H, hd, float(base), posOffset, ex.data, eo.data))
        if needs:
            eo.ropeOf = (x, ex, H, hd, base, posOffset)

        return self._record(out, needs, self._ropeBackward, x, ex, eo, T, H, hd, base, posOffset)

    def _ropeBackward(self, x, ex, eo, T, H, hd, base, posOffset):
        self._ensureBackwardBegun()
        if eo.ropeFused and not (eo.gradLive or eo.copyFrom or eo.pendingDx is not None):
            return                       # attention's backward already delivered this gradient to x
        go = self._gradSource(eo)
        gx, ax = self._gradTarget(x, ex)
        self._check(self.lib.gt_rope_bwd(self.ctx, T, H, hd, float(base), posOffset, go, gx, ax))

    def attention(self, q: Tensor, k: Tensor, v: Tensor, T: int, Hq: int, Hkv: int, hd: int, window: int) -> Tensor:
        """webgpu.ts:1125-1192."""
        self._beginForwardOp()
        self._checkT(T, q.shape[0], "attention")
        eq, ek, ev = self._entryFor(q), self._entryFor(k), self._entryFor(v)
        needs = self._flows(q, eq) or self._flows(k, ek) or self._flows(v, ev)
        rec = self._curRec
        nbytes = T * Hq * hd * 4
        if rec is not None and rec["replay"] and rec["pos"] < len(rec["saved"]) and rec["saved"][rec["pos"]][2] == nbytes:
            # replay of a recompute region: the first run's output and row statistics, no launch
            data, lse, _n = rec["saved"][rec["pos"]]
            rec["pos"] += 1
            out = Tensor.output([T, Hq * hd], T * Hq * hd, [q, k, v])
            eo = _entry(self._uid, data, nbytes, out.size)
            eo.needs, eo.region = needs, self._regionStack[-1][0]
            out._needs, out._dev = needs, eo
        else:
            out, eo = self._makeOut([T, Hq * hd], T * Hq * hd, [q, k, v], needs)
            lse = self._acquireRecycled(Hq * T * 4)
            self._check(self.lib.gt_attention_fwd(self.ctx, T, Hq, Hkv, hd, window, eq.data, ek.data, ev.data, eo.data, lse))
            if rec is not None and not rec["replay"]:
                rec["saved"].append((eo.data, lse, nbytes))

        return self._record(out, needs, self._attentionBackward, q, eq, k, ek, v, ev, eo, lse, T, Hq, Hkv, hd, window)

    def _attentionBackward(self, q, eq, k, ek, v, ev, eo, lse, T, Hq, Hkv, hd, window):
        self._ensureBackwardBegun()
        go = self._gradSource(eo)
        rq, rk = eq.ropeOf, ek.ropeOf
        fresh = lambda e: not (e.gradLive or e.copyFrom or e.pendingDx is not None)
        if (self.fuseRope and rq is not None and rk is not None and eq is not ek and rq[3:] == rk[3:] and rq[3] == hd
                and rq[2] == Hq and rk[2] == Hkv and hd in (64, 128) and T >= 64 and self.precision == "tf32"
                and fresh(eq) and fresh(ek)):
            # q and k came out of rotary embeddings and nothing else has written their gradients: the kernels rotate
            # dQ and dK back as they store them, into the gradients of the embeddings' inputs
            gq, aq = self._gradTarget(rq[0], rq[1])
            gk, ak = self._gradTarget(rk[0], rk[1])
            gv, av = self._gradTarget(v, ev)
            self._check(self.lib.gt_attention_bwd_rope(self.ctx, T, Hq, Hkv, hd, window, eq.data, ek.data, ev.data, eo.data,
                                                       lse, go, gq, aq, gk, ak, gv, av, float(rq[4]), rq[5]))
            eq.ropeFused = ek.ropeFused = True
            return
        gq, aq = self._gradTarget(q, eq)
        gk, ak = self._gradTarget(k, ek)
        gv, av = self._gradTarget(v, ev)
        self._check(self.lib.gt_attention_bwd(self.ctx, T, Hq, Hkv, hd, window, eq.data, ek.data, ev.data, eo.data,
                                              lse, go, gq, aq, gk, ak, gv, av))

    def _nseq(self) -> int:
        return self._batch[0] if self._batch[0] else 1

    def _lossOut(self, prev, needs: bool):
        """The scalar loss tensor plus its device-side companions: [1+nseq] losses and [nseq] 1/kept."""
        nseq = self._nseq()
        loss = Tensor.output([1], 1, list(prev))
        e = _entry(self._uid, self._acquireRecycled((1 + nseq) * 4), 4, 1)
        e.needs = loss._needs = needs
        e.region = self._regionStack[-1][0] if self._regionStack else 0
        loss._dev = e
        invKept = self._acquireRecycled(nseq * 4)
        return loss, e, invKept

    def _lossGrad(self, loss: Tensor, e: _Entry) -> int:
        """backward(loss, seed) wrote the seed into the HOST grad array; push it to the device
        (webgpu.ts:1316-1320). A captured graph instead reads the seed from a fixed buffer that
        beginCapture filled, since a host write cannot be replayed."""
        if self._capturing:
            return self._seedBuf
        if not e.gradLive:
            self._write(self._gradAddr(e), loss.grad[:1])
            e.gradLive = True
        return e.grad

    def crossEntropy(self, logits: Tensor, targets, kept: int) -> Tensor:
        """webgpu.ts:1295-1329. `kept` was counted above the dispatch; the device derives the same
        count from the uploaded targets, so nothing host-computed is baked into a replayable graph."""
        # The readout that makes the logits usually waits to be launched: then it takes the loss's statistics as it writes them.
        readout = None
        fused = getattr(self.lib, "gt_readout_ce_fwd", None)    # (a stand-in for the library need not have it)
        pend = self._pendingFwd
        if (fused is not None and len(pend) == 1 and logits._dev is pend[0]["eo"] and logits._dev.owner == self._uid
                and not ("rope" in pend[0] or "lora" in pend[0] or "norm" in pend[0])):
            readout = pend[0]
        self._beginForwardOp(keepPending=readout is not None)
        T, V = logits.shape
        tgt = self._uploadU32(targets, "targets", V)
        if readout is not None:
            self._pendingFwd = []
            readout["eo"].pendingFwd = False
        el = self._entryFor(logits)
        stats = self._acquireRecycled(T * 16)
        needs = self._flows(logits, el)
        loss, eo, invKept = self._lossOut([logits], needs)
        if readout is not None:
            self._check(fused(self.ctx, T, V, readout["inDim"], readout["ex"].data, readout["ew"].data, el.data, tgt, stats, eo.data, invKept))
        else:
            self._check(self.lib.gt_ce_fwd(self.ctx, T, V, el.data, tgt, stats, eo.data, invKept))

        def _bw():
            self._ensureBackwardBegun()
            seed = self._lossGrad(loss, eo)
            gl, al = self._gradTarget(logits, el)
            self._check(self.lib.gt_ce_bwd(self.ctx, T, V, el.data, tgt, stats, invKept, seed, gl, al))

        return self._record(loss, needs, _bw)

    def fusedCrossEntropy(self, hidden: Tensor, w: Tensor, targets, chunk: int, kept: int) -> Tensor:
        """webgpu.ts:1214-1278: per vocab span, logits = hidden·W[span]ᵀ then online (max, sum, target
        logit); backward recomputes each span, forms dlogits in place and feeds the two products."""
        self._beginForwardOp()
        T, H = hidden.shape
        V = w.shape[0]
        eh, ew = self._entryFor(hidden), self._entryFor(w)
        tgt = self._uploadU32(targets, "targets", V)
        run = self._acquireRecycled(T * 12)
        width = min(chunk, V)
        ch = self._acquireRecycled(T * width * 4)
        needs = self._flows(hidden, eh) or self._flows(w, ew)
        loss, eo, invKept = self._lossOut([hidden, w], needs)
        # the product of a span with its statistics or its gradient in one call (a library without these makes two of it)
        fusedStats, fusedGrad = (getattr(self.lib, name, None) for name in ("gt_readout_ce_stats", "gt_readout_ce_grad"))
        for v0 in range(0, V, chunk):
            n = min(chunk, V - v0)
            if fusedStats is not None:
                self._check(fusedStats(self.ctx, T, n, H, v0, 1 if v0 == 0 else 0, eh.data, ew.data + v0 * H * 4, ch, tgt, run))
            else:
                self._gemm("NT", 0, T, n, H, eh.data, ew.data + v0 * H * 4, ch)
                self._check(self.lib.gt_ce_chunk_stats(self.ctx, T, n, v0, 1 if v0 == 0 else 0, ch, tgt, run))
        self._check(self.lib.gt_ce_loss_from_stats(self.ctx, T, run, tgt, eo.data, invKept))

        def _bw():
            self._ensureBackwardBegun()
            seed = self._lossGrad(loss, eo)
            gh, ah = self._gradTarget(hidden, eh)
            gw, aw = self._gradTarget(w, ew)
            for v0 in range(0, V, chunk):
                n = min(chunk, V - v0)
                if fusedGrad is not None:
                    self._check(fusedGrad(self.ctx, T, n, H, v0, eh.data, ew.data + v0 * H * 4, ch, tgt, run, invKept, seed))
                else:
                    self._gemm("NT", 0, T, n, H, eh.data, ew.data + v0 * H * 4, ch)
                    self._check(self.lib.gt_ce_chunk_grad(self.ctx, T, n, v0, ch, tgt, run, invKept, seed))
                if gh:
                    self._gemm("NN", ah, T, H, n, ch, ew.data + v0 * H * 4, gh)
                    ah = 1
                if gw:
                    # rows [v0, v0+n) of dW; each span is written by exactly one product
                    self._gemm("TN", aw, n, H, T, ch, eh.data, gw + v0 * H * 4)

        return self._record(loss, needs, _bw)

    def softCrossEntropy(self, logits: Tensor, teacherIds, teacherProbs, k: int, kept: int) -> Tensor:
        """webgpu.ts:1331-1378."""
        self._beginForwardOp()
        T, V = logits.shape
        el = self._entryFor(logits)
        ids = self._uploadU32(teacherIds, "teacher", V)
        probs = self._uploadF32(teacherProbs)
        stats = self._acquireRecycled(T * 16)
        needs = self._flows(logits, el)
        loss, eo, invKept = self._lossOut([logits], needs)
        self._check(self.lib.gt_soft_ce_fwd(self.ctx, T, V, k, el.data, ids, probs, stats, eo.data, invKept))

        def _bw():
            self._ensureBackwardBegun()
            seed = self._lossGrad(loss, eo)
            gl, al = self._gradTarget(logits, el)
            self._check(self.lib.gt_soft_ce_bwd(self.ctx, T, V, k, el.data, ids, probs, stats, invKept, seed, gl, al))

        return self._record(loss, needs, _bw)

    # ------------------------------------------------------------------ per-sequence losses of a batched call
    def sequenceLosses(self, loss: Tensor) -> np.ndarray:
        """The per-sequence losses behind a loss tensor produced under setBatch (blocks)."""
        e = self._entries[loss]
        out = np.empty(1 + self._nseq(), np.float32)
        self._read(e.data, out)
        return out[1:]


def _destroy_ctx(lib, ctx):
    try:
        lib.gt_destroy(ctx)
    except Exception:
        pass


def initCuda(device: int = 0, precision: str = "fp32") -> Optional[CudaBackend]:
    """`initWebGPU()` (webgpu.ts:1812-1870): a backend, or None when there is no GPU so suites can SKIP."""
    try:
        return CudaBackend(device, precision)
    except _lib.GtError:
        return None


def requireGPU(purpose: str, device: int = 0, precision: str = "fp32") -> CudaBackend:
    """webgpu.ts:1872-1888."""
    gpu = initCuda(device, precision)
    if gpu is None:
        raise RuntimeError(f"no GPU adapter found, and {purpose} needs one")
    return gpu
