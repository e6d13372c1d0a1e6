"""Tensor-level wrappers over the C ABI: allocate outputs with torch, pass raw pointers and the current stream.

Every operator of the package goes through the object returned by :func:`get_backend`.  The only
back end is :class:`CudaBackend`; it refuses tensors that are not on a CUDA device, and constructing it
raises if ``libmlcg_b200.so`` is missing.
"""
import contextlib
import ctypes
import threading
from dataclasses import dataclass
from typing import Optional

import numpy as np
import torch

from . import _lib

_DT = {torch.float32: 0, torch.float64: 1}
STATUS_TRUNCATED, STATUS_BAD_INDEX, STATUS_ASYMMETRIC, STATUS_NOT_THERE, STATUS_SIZES = 1, 2, 4, 64, 128


@dataclass(frozen=True)
class RbfSpec:
    """Host-side description of a radial basis x envelope (mirror of ``mlcgb_rbf_spec``)."""

    kind: int          # 0 Gaussian, 1 exp-normal
    num_rbf: int
    cutoff_kind: int   # 0 identity, 1 cosine
    lower: float
    upper: float
    alpha: float
    p0: torch.Tensor   # offsets | means
    p1: torch.Tensor   # coeff (1 element) | betas


class _WeightPlaces:
    """Where the gradient of each packed weight lies in one flat buffer, in the order of the weights."""

    def __init__(self, tensors):
        self.total, at = 0, []
        for k, t in enumerate(tensors):
            if t is None or k == 4:
                at.append(-1)
            else:
                at.append(4 * self.total)
                self.total += t.numel()
        self.head = at[:4]
        self.blocks = (ctypes.c_int64 * (len(at) - 5))(*at[5:])
        self.blocks = np.frombuffer(self.blocks, dtype=np.int64)          # (every weight of a block is there)

    def struct(self, w, base):
        addresses = self.blocks + base
        arr = (_lib.SchnetBlockStruct * w.num_blocks).from_buffer(addresses)
        return _lib.SchnetWeightsStruct(w.hidden, w.filters, w.conv_out, w.head_width, w.num_blocks, w.num_types, arr,
                                        *(None if h < 0 else base + h for h in self.head), None), addresses


def weights_struct(sizes, tensors):
    """``mlcgb_schnet_weights`` over ``tensors`` (in the packed order; None: absent) with the widths and counts of ``sizes``, another such
    structure or anything with its fields, and the block array it points to."""
    ptr = [None if t is None else t.data_ptr() for t in tensors]
    arr = (_lib.SchnetBlockStruct * sizes.num_blocks)(*(_lib.SchnetBlockStruct(*ptr[k: k + 8]) for k in range(5, len(ptr), 8)))
    return _lib.SchnetWeightsStruct(sizes.hidden, sizes.filters, sizes.conv_out, sizes.head_width, sizes.num_blocks, sizes.num_types, arr, *ptr[:5]), arr


def _weights_places(weights):
    struct, (_, tensors, *_) = weights
    places = struct.__dict__.get("places")
    if places is None:
        places = struct.places = _WeightPlaces(tensors)
    return places


class ForceMatchingState:
    """What the backward of a force-matching step needs of its forward pass.  ``tensors``: the device buffers, which the pass's autograd
    node takes over as saved tensors; everything else says where in them things lie.  No address outlives the forward pass: saved-tensor
    hooks may bring the buffers back elsewhere.  ``places``: (index in ``tensors``, byte offset) of each of :attr:`NAMES`."""

    NAMES = ("types", "struct_ptr", "row0", "row1", "offsets", "sel", "pair_of", "forward_ws", "twin", "p0", "p1")
    __slots__ = ("N", "B", "E", "tensors", "places", "spec", "conv_cut", "weights")

    def __init__(self, *values):
        self.N, self.B, self.E, self.tensors, self.places, self.spec, self.conv_cut, self.weights = values

    def addresses(self, saved):
        base = [0 if t is None else t.data_ptr() for t in saved]
        return [base[k] + at for k, at in self.places]

    def view(self, saved, name):
        k, at = self.places[self.NAMES.index(name)]
        if saved[k].dtype != torch.uint8:             # (a tensor of its own)
            return saved[k]
        entries, dtype = {"struct_ptr": (self.B + 1, torch.int64), "offsets": (self.N + 1, torch.int64), "sel": (self.E // 2, torch.int32),
                          "forward_ws": (3 * self.N, torch.float32)}.get(name, (self.E, torch.int32))
        return saved[k][at: at + entries * dtype.itemsize].view(dtype)

    def positions(self, saved):
        return self.view(saved, "forward_ws").view(self.N, 3)


def _ptr(t: Optional[torch.Tensor]):
    return None if t is None else t.data_ptr()


def _stream():
    """Raw handle of torch's current stream on the current device."""
    return torch._C._cuda_getCurrentRawStream(torch._C._cuda_getDevice())


class _NoGuard:
    def __enter__(self):
        return None

    def __exit__(self, *exc):
        return False


_NO_GUARD = _NoGuard()


@contextlib.contextmanager
def _outside_inference():
    with torch.inference_mode(False), torch.no_grad():
        yield


def lasting():
    """The mode in which what is kept for later calls is made, whatever the caller's: a tensor made under ``torch.inference_mode()`` has no
    count of the writes to it and can enter no graph outside."""
    return _outside_inference() if torch.is_inference_mode_enabled() else _NO_GUARD


def _on(device):
    """Device guard for a launch: a real ``torch.cuda.device`` only when ``device`` is not the current one."""
    if device.index is None or device.index == torch._C._cuda_getDevice():
        return _NO_GUARD
    return torch.cuda.device(device)


def _need_cuda(*ts):
    """Every tensor whose address a kernel gets is on the device of the first one."""
    device = None
    for t in ts:
        if t is None:
            continue
        if not t.is_cuda:
            raise RuntimeError("mlcg_b200 operators run on CUDA tensors only (there is no CPU fallback)")
        if device is None:
            device = t.get_device()
        elif t.get_device() != device:
            raise RuntimeError(f"mlcg_b200: tensors on different devices (cuda:{device} and {t.device})")


def _raise_for_status(word: int, what: str) -> None:
    """Status bits the tensor-core kernels set (read lazily, with the next unavoidable host read)."""
    if word & STATUS_SIZES:
        raise ValueError(f"mlcg_b200: {what}: n_atoms does not add up to the positions")
    if word & 8:
        raise RuntimeError(f"mlcg_b200: {what}: a tensor-core wait ran out; results are incomplete")
    if word & 32:
        raise RuntimeError(f"mlcg_b200: {what}: the radius graph has more edges than the fixed edge capacity; results are incomplete "
                           "(raise the capacity)")
    if word & 4:
        raise RuntimeError(f"mlcg_b200: {what}: the edge list is not symmetric (an edge without its reverse, e.g. after the neighbour "
                           "cap cut a list short)")
    if word & 16:
        raise RuntimeError(f"mlcg_b200: {what}: a weight is beyond the range of the fp16-pair tensor-core operands (|w| > 512); "
                           "set mlcg_b200.backend.get_backend().tensor_core_gemm = False to run these layers on the CUDA cores")


def _dt(t: torch.Tensor) -> int:
    try:
        return _DT[t.dtype]
    except KeyError:
        raise TypeError(f"mlcg_b200: unsupported dtype {t.dtype}; use float32 or float64") from None


class KernelProfiler:
    """Per-operator launch counts, device time (CUDA events on the launching stream) and algorithmic work.

    Attach with ``get_backend().profiler = KernelProfiler()``; ``summary()`` synchronises and returns
    ``{name: {"calls", "launches", "ms", "bytes", "flops"}}``."""

    def __init__(self, time_kernels: bool = True):
        self.time_kernels = time_kernels
        self.records = []      # (name, start_event, end_event)
        self.stats = {}

    def begin(self, name, launches, nbytes, flops):
        st = self.stats.setdefault(name, {"calls": 0, "launches": 0, "ms": 0.0, "bytes": 0, "flops": 0})
        st["calls"] += 1
        st["launches"] += launches
        st["bytes"] += int(nbytes)
        st["flops"] += int(flops)
        if not self.time_kernels:
            return None
        ev = torch.cuda.Event(enable_timing=True)
        ev.record()
        return ev

    def end(self, name, start):
        if start is None:
            return
        ev = torch.cuda.Event(enable_timing=True)
        ev.record()
        self.records.append((name, start, ev))

    def summary(self):
        torch.cuda.synchronize()
        for name, a, b in self.records:
            self.stats[name]["ms"] += a.elapsed_time(b)
        self.records = []
        return self.stats

    @property
    def total_launches(self):
        return sum(v["launches"] for v in self.stats.values())


class _Lists(threading.local):
    made = 0            # prior lists prepared by this thread
    word = None         # the status word behind the last of them, where its call has waited


class CudaBackend:
    name = "cuda"

    def __init__(self):
        self.lib = _lib.load()
        _lib.bind_native(self.lib)
        self.native = _lib.native()
        self.profiler = None
        self._status, self.lists = {}, _Lists()
        self.tensor_core_gemm = True   # float32 GEMMs of qualifying shape run on tcgen05 (fp32-equivalent products)
        self._pending = []      # (status tensor, what) of kernels whose status word has not been read yet

    def defer_status(self, status, what):
        """Remember a kernel's status word; it is read together with the next unavoidable host read (the edge
        count of the next radius graph) or by :meth:`check_pending`, so the hot path gains no synchronisation."""
        if not self._pending or (self._pending[-1][0] is not status and not any(s is status for s, _ in self._pending)):
            self._pending.append((status, what))
        if len(self._pending) > 256:
            self.check_pending()

    def check_pending(self):
        pending, self._pending = self._pending, []
        if not pending:
            return
        words = [0] * len(pending)
        for dev in {s.device for s, _ in pending}:         # one read per device
            here = [k for k, (s, _) in enumerate(pending) if s.device == dev]
            for k, word in zip(here, torch.stack([pending[k][0][0] for k in here]).cpu().tolist()):
                words[k] = word
        self._raise_pending(words, pending)

    def _take_pending(self, dev):
        """The one status word that waits to be read, for a kernel on ``dev`` to hand over with its own result; more than one, or one of
        another device, are read here."""
        if len(self._pending) > 1 or (self._pending and self._pending[0][0].device != dev):
            self.check_pending()
        pend, self._pending = self._pending, []
        return pend

    @staticmethod
    def _raise_pending(words, pending):
        """Raise for the first status word that reports a failure; the words are cleared first, so one failure is reported
        once and later evaluations start clean."""
        bad = [(w, what) for w, (_, what) in zip(words, pending) if w & (4 | 8 | 16 | 32 | STATUS_SIZES)]
        if bad:
            for st, _ in pending:
                st.zero_()
            _raise_for_status(*bad[0])

    # ------------------------------------------------------------------ device time per entry point
    def timeline_begin(self):
        """Start recording a CUDA event pair around every kernel-launching library call made from this thread."""
        _lib.check(self.lib.mlcgb_timeline_begin(), "timeline_begin")

    def timeline_end(self):
        """Stop recording, wait for the events and return ``{entry point: {"calls": n, "ms": total}}``."""
        n = self.lib.mlcgb_timeline_end()
        if n < 0:
            _lib.check(n, "timeline_end")
        out = {}
        name, calls, ms = ctypes.c_char_p(), ctypes.c_int64(), ctypes.c_double()
        for i in range(n):
            _lib.check(self.lib.mlcgb_timeline_entry(i, ctypes.byref(name), ctypes.byref(calls), ctypes.byref(ms)), "timeline_entry")
            out[name.value.decode()] = {"calls": int(calls.value), "ms": float(ms.value)}
        return out

    def _run(self, name, fn, args, what=None, launches=1, nbytes=0, flops=0):
        prof = self.profiler
        ev = prof.begin(name, launches, nbytes, flops) if prof is not None else None
        _lib.check(fn(*args), what or name)
        if prof is not None:
            prof.end(name, ev)

    def _work(self, name, v):
        """Algorithmic bytes / flops and kernel launches of one call (index tensors counted at their stored width); only
        worked out while a profiler is attached."""
        if self.profiler is None:
            return {}
        es = lambda t: t.element_size()
        if name == "radius_count":
            return dict(launches=5, nbytes=v["N"] * (12 + 4 + 8) + v["B"] * 8)
        if name == "radius_fill":
            return dict(launches=1, nbytes=16 * v["E"] + 20 * v["N"])       # [2,E] int64 written, pos + structure ids read
        if name == "seg_mul_sum":
            V, a = v["V"], v["a"]
            return dict(nbytes=V.numel() * es(V) + V.shape[0] * 4 + (a.numel() + v["N"] * v["F"]) * es(V) + v["N"] * 8,
                        flops=2 * V.numel())
        if name == "edge_mul":
            a = v["a"]
            return dict(nbytes=v["E"] * v["F"] * es(a) + v["E"] * 8 + 2 * a.numel() * es(a), flops=v["E"] * v["F"])
        if name == "gemm":
            A = v["A"]
            M, N, K = v["M"], v["N"], v["K"]
            return dict(launches=2 if v["wsb"] else 1, nbytes=(M * K + N * K + M * N) * es(A), flops=2 * M * N * K)
        if name in ("rbf_expand", "rbf_contract"):
            d = v["d"]
            R = v["spec"].num_rbf
            return dict(nbytes=d.numel() * es(d) * (R + 1 + (1 if name == "rbf_contract" else 0)), flops=d.numel() * R * 20)
        if name == "edge_diff":
            return dict(nbytes=v["E"] * (8 + 3 * es(v["pos"])) + v["pos"].numel() * es(v["pos"]))
        if name == "node_scatter_diff":
            g = v["g"]
            return dict(nbytes=2 * g.numel() * es(g) + g.shape[0] * 4 + v["N"] * (16 + 3 * es(g)))
        if name == "prior_terms":
            m = v["mapping"]
            return dict(nbytes=m.numel() * 8 + v["M"] * 8 + v["params"].numel() * es(v["params"]) + 2 * v["pos"].numel() * es(v["pos"]))
        return {}

    # ------------------------------------------------------------------ radius graph
    def batch_to_ptr(self, batch: torch.Tensor, B: int) -> torch.Tensor:
        _need_cuda(batch)
        batch = batch.contiguous()
        ptr = torch.empty(B + 1, dtype=torch.int64, device=batch.device)
        with _on(batch.device):
            self._run("batch_to_ptr", self.lib.mlcgb_batch_to_ptr, (_ptr(batch), batch.numel(), B, _ptr(ptr), _stream(),), **self._work("batch_to_ptr", locals()))
        return ptr

    def batch_boundaries(self, batch: torch.Tensor) -> torch.Tensor:
        """The boundaries of the ``int(batch[-1]) + 1`` structures of a sorted int64 batch vector."""
        _need_cuda(batch)
        batch = batch.contiguous()
        N, host = batch.numel(), ctypes.c_int64()
        ptr = torch.empty(N + 1, dtype=torch.int64, device=batch.device)
        with _on(batch.device):
            _lib.check(self.lib.mlcgb_batch_boundaries(_ptr(batch), N, N, _ptr(ptr), ctypes.addressof(host), _stream()), "batch_boundaries")
        B = host.value
        return ptr[:B + 1] if 0 <= B <= N else self.batch_to_ptr(batch, B)

    def radius_graph(self, pos, ptr, r, max_num_neighbors, loop, rule, want_distance=False, want_batch=True, exclude=None, n_atoms=None, want_index=True,
                     want_plan=False, want_rows=True):
        """Returns dict(edge_index[2,E] i64, distance|None, mapping_batch|None, row0, row1 (i32), offsets[N+1] i64, status int).
        ``exclude``: ``(exclude_pair_xs, ptr_exclude_pair_xs)`` int64 as ``mlcg::radius_cuda`` takes them (rule "native" only).
        ``n_atoms`` (int64 [B] on the device) in place of ``ptr`` (None then; the boundaries come back under ``"ptr"``).
        ``want_plan``: also twin, sel and pair_of as :meth:`pair_plan` gives them, or None under these keys where a list was cut short,
        has loops or exclusions, or has no edges; ``want_index=False``: no int64 edge index; ``want_rows=False`` (an index and no plan
        then): None for row0 and row1."""
        _need_cuda(pos, ptr, n_atoms)
        ptr, n_atoms = (None if t is None else t.contiguous() for t in (ptr, n_atoms))
        ex_xs = ex_ptr = None
        if exclude is not None:
            if int(rule) != 0:
                raise ValueError("excluded pairs go with the neighbour cap of radius.cu (rule 0)")
            ex_xs, ex_ptr = (t.to(device=pos.device, dtype=torch.int64).contiguous() for t in exclude)
            if ex_ptr.numel() != pos.shape[0] + 1:
                raise ValueError("ptr_exclude_pair_xs must have one entry per point plus one")
        pos = pos.detach().contiguous()
        N, dev = pos.shape[0], pos.device
        B = ptr.numel() - 1 if n_atoms is None else n_atoms.numel()
        dt, loop = _dt(pos), int(bool(loop))
        with _on(dev):
            if ptr is None:
                ptr = torch.empty(B + 1, dtype=torch.int64, device=dev)
            if N == 0 or B == 0:
                if n_atoms is not None:
                    ptr.zero_()
                empty = torch.empty(0, dtype=torch.int32, device=dev)
                return dict(edge_index=torch.empty((2, 0), dtype=torch.int64, device=dev), distance=pos.new_empty(0) if want_distance else None,
                            mapping_batch=torch.empty(0, dtype=torch.int64, device=dev) if want_batch else None, row0=empty, row1=empty.clone(),
                            offsets=torch.zeros(N + 1, dtype=torch.int64, device=dev), status=0, ptr=ptr, twin=None, sel=None, pair_of=None)
            pend = self._take_pending(dev)
            wsb = self.lib.mlcgb_graph_workspace_bytes(N, B, dt)
            ws = torch.empty(wsb, dtype=torch.uint8, device=dev)
            offsets = torch.empty(N + 1, dtype=torch.int64, device=dev)
            host = (ctypes.c_int64 * 4)()
            common = (_ptr(pos), dt)
            self._run("radius_count", self.lib.mlcgb_graph_begin, common + (
                _ptr(n_atoms), _ptr(ptr), N, B, float(r), int(max_num_neighbors), loop, int(rule), _ptr(ex_xs), _ptr(ex_ptr), _ptr(ws), wsb,
                _ptr(offsets), _ptr(pend[0][0]) if pend else None, host, _stream()), **self._work("radius_count", locals()))   # the one host read
            E, st = host[0], int(host[1])
            if pend and host[2]:
                self._raise_pending([int(host[2])], pend)
            if st & STATUS_SIZES:
                _raise_for_status(st, "radius graph")
            plan = want_plan and not loop and exclude is None and not st & STATUS_TRUNCATED and 0 < E < 1 << 31 and E % 2 == 0
            ei = torch.empty((2, E), dtype=torch.int64, device=dev) if want_index else None
            dist = torch.empty(E, dtype=pos.dtype, device=dev) if want_distance else None
            mb = torch.empty(E, dtype=torch.int64, device=dev) if want_batch else None
            twin = sel = pair_of = None
            if plan:
                pad = -E % 8        # (row1 on a 32-byte boundary)
                r0, _, r1, twin, pair_of, sel = torch.empty(4 * E + pad + E // 2, dtype=torch.int32, device=dev).split((E, pad, E, E, E, E // 2))
            else:
                r0, r1 = torch.empty(2 * E, dtype=torch.int32, device=dev).split((E, E)) if want_rows else (None, None)
            self._run("radius_fill", self.lib.mlcgb_graph_finish, common + (
                _ptr(ptr), N, B, float(r), loop, _ptr(ex_xs), _ptr(ex_ptr), _ptr(ws), wsb, _ptr(offsets), E, _ptr(ei), _ptr(dist), _ptr(mb), _ptr(r0),
                _ptr(r1), _ptr(twin), _ptr(sel), _ptr(pair_of), int(host[3] != 0), _ptr(self._sticky_status(dev)), _stream()), **self._work("radius_fill", locals()))
        return dict(edge_index=ei, distance=dist, mapping_batch=mb, row0=r0, row1=r1, offsets=offsets, status=st, ptr=ptr, twin=twin, sel=sel,
                    pair_of=pair_of)

    small_graph_points = 2048       # what mlcgb_graph_small_begin takes

    def radius_graph_small(self, pos, batch, r, max_num_neighbors, loop, rule, want_distance=False):
        """:meth:`radius_graph` of 1 to 2048 points with their sorted batch vector (int64; None: one structure): edge_index, distance,
        offsets and status, nothing else."""
        _need_cuda(pos, batch)
        batch = None if batch is None else batch.contiguous()
        pos = pos.detach().contiguous()
        N, dev = pos.shape[0], pos.device
        dt, loop = _dt(pos), int(bool(loop))
        with _on(dev):
            pend = self._take_pending(dev)
            wsb = self.lib.mlcgb_graph_workspace_bytes(N, 1, dt)
            ws = torch.empty(wsb, dtype=torch.uint8, device=dev)
            offsets = torch.empty(N + 1, dtype=torch.int64, device=dev)
            host = (ctypes.c_int64 * 4)()
            self._run("radius_count", self.lib.mlcgb_graph_small_begin, (
                _ptr(pos), dt, _ptr(batch), N, float(r), int(max_num_neighbors), loop, int(rule), _ptr(ws), wsb, _ptr(offsets),
                _ptr(pend[0][0]) if pend else None, host, _stream()))
            E = host[0]
            if pend and host[2]:
                self._raise_pending([int(host[2])], pend)
            ei = torch.empty((2, E), dtype=torch.int64, device=dev)
            dist = torch.empty(E, dtype=pos.dtype, device=dev) if want_distance else None
            self._run("radius_fill", self.lib.mlcgb_graph_small_finish, (_ptr(pos), dt, _ptr(batch), N, _ptr(ws), wsb, _ptr(offsets), E, _ptr(ei), _ptr(dist),
                                                                         _stream()))
        return dict(edge_index=ei, distance=dist, offsets=offsets, status=int(host[1]))

    def radius_graph_pbc(self, pos, ptr, cells, repeats, r, max_num_neighbors, loop, want_distance=False, want_batch=True):
        """Radius graph of periodic structures: dict(edge_index [2,E] i64 (row 0 = centre), cell_shifts [E,3], distance|None,
        mapping_batch|None, status int).  ``cells`` [B,3,3] in the dtype of ``pos``, ``repeats`` [B,3] copies per cell vector."""
        _need_cuda(pos, ptr, cells, repeats)
        pos, ptr = pos.detach().contiguous(), ptr.contiguous()
        cells = cells.detach().to(pos.dtype).contiguous()
        repeats = repeats.to(torch.int32).contiguous()
        N, B, dev = pos.shape[0], ptr.numel() - 1, pos.device
        if cells.numel() != 9 * B or repeats.numel() != 3 * B:
            raise ValueError("cells must be [B,3,3] and repeats [B,3]")
        dt = _dt(pos)
        with _on(dev):
            wsb = self.lib.mlcgb_radius_pbc_workspace_bytes(N)
            ws = torch.empty(max(wsb, 1), dtype=torch.uint8, device=dev)
            deg = torch.empty(max(N, 1), dtype=torch.int32, device=dev)
            offsets = torch.empty(N + 1, dtype=torch.int64, device=dev)
            status = torch.zeros(4, dtype=torch.int32, device=dev)
            self._run("radius_pbc_count", self.lib.mlcgb_radius_pbc_count,
                      (_ptr(pos), dt, _ptr(ptr), N, B, _ptr(cells), _ptr(repeats), float(r), int(max_num_neighbors), int(loop), _ptr(ws), wsb,
                       _ptr(deg), _ptr(offsets), _ptr(status), _stream()), launches=5)
            E, st = (int(v) for v in torch.stack([offsets[N], status[0].to(torch.int64)]).cpu().tolist())
            ei = torch.empty((2, E), dtype=torch.int64, device=dev)
            shifts = torch.empty((E, 3), dtype=pos.dtype, device=dev)
            dist = torch.empty(E, dtype=pos.dtype, device=dev) if want_distance else None
            mb = torch.empty(E, dtype=torch.int64, device=dev) if want_batch else None
            self._run("radius_pbc_fill", self.lib.mlcgb_radius_pbc_fill,
                      (_ptr(pos), dt, _ptr(ptr), N, B, _ptr(cells), _ptr(repeats), float(r), int(max_num_neighbors), int(loop), _ptr(ws), wsb,
                       _ptr(offsets), E, _ptr(ei), _ptr(shifts), _ptr(dist), _ptr(mb), _ptr(status), _stream()), nbytes=E * (16 + 3 * pos.element_size()))
        return dict(edge_index=ei, cell_shifts=shifts, distance=dist, mapping_batch=mb, offsets=offsets, status=st)

    def radius_graph_capacity(self, pos, ptr, r, max_num_neighbors, capacity, rows=None, rule=1):
        """The radius graph into buffers of ``capacity`` edges without reading the edge count on the host:
        dict(row0, row1 (int32 [capacity]), offsets [N+1], counts (int64 [2] on the device: edges, edges / 2)).  ``rows``: an int32
        ``[2, capacity]`` buffer to reuse, whose entries are valid point indices (zeros at first).  An overflow sets bit 5 of the
        backend's accumulating status words (reported by :meth:`check_pending`)."""
        _need_cuda(pos, ptr)
        pos, ptr = pos.detach().contiguous(), ptr.contiguous()
        N, B, dev = pos.shape[0], ptr.numel() - 1, pos.device
        dt = _dt(pos)
        capacity = int(capacity)
        if capacity < 0 or capacity % 2:
            raise ValueError("capacity must be a non-negative even number of edges")
        if rows is None:
            rows = torch.zeros((2, capacity), dtype=torch.int32, device=dev)
        with _on(dev):
            ws_bytes = self.lib.mlcgb_radius_workspace_bytes(N, B, dt)
            ws = torch.empty(max(ws_bytes, 1), dtype=torch.uint8, device=dev)
            deg = torch.empty(max(N, 1), dtype=torch.int32, device=dev)
            offsets = torch.empty(N + 1, dtype=torch.int64, device=dev)
            counts = torch.empty(2, dtype=torch.int64, device=dev)
            status = self._sticky_status(dev)
            self._run("radius_graph_capacity", self.lib.mlcgb_radius_graph_capacity,
                      (_ptr(pos), dt, _ptr(ptr), N, B, float(r), int(max_num_neighbors), 0, int(rule), _ptr(ws), ws_bytes, _ptr(deg), _ptr(offsets),
                       capacity, None, _ptr(rows[0]), _ptr(rows[1]), _ptr(counts), _ptr(status), _stream()), launches=7, nbytes=N * 24 + capacity * 8)
        self.defer_status(status, "radius graph with a fixed edge capacity")
        return dict(row0=rows[0], row1=rows[1], offsets=offsets, counts=counts)

    def graph_capacity(self, pos, ptr, n_atoms, r, max_num_neighbors, capacity, rows, rule=1):
        """:meth:`radius_graph_capacity` and :meth:`pair_plan` together, from ``n_atoms`` (int64 [B]; ``ptr`` None) or ``ptr``:
        dict(row0, row1, offsets, counts, ptr, twin, sel, pair_of)."""
        _need_cuda(pos, ptr, n_atoms)
        ptr, n_atoms = (None if t is None else t.contiguous() for t in (ptr, n_atoms))
        pos = pos.detach().contiguous()
        N, dev, dt = pos.shape[0], pos.device, _dt(pos)
        B = ptr.numel() - 1 if n_atoms is None else n_atoms.numel()
        capacity = int(capacity)
        if capacity < 0 or capacity % 2:
            raise ValueError("capacity must be a non-negative even number of edges")
        with _on(dev):
            if ptr is None:
                ptr = torch.empty(B + 1, dtype=torch.int64, device=dev)
            wsb = self.lib.mlcgb_graph_workspace_bytes(N, B, dt)
            ws = torch.empty(wsb, dtype=torch.uint8, device=dev)
            offsets, counts = torch.empty(N + 3, dtype=torch.int64, device=dev).split((N + 1, 2))
            twin, pair_of, sel = torch.empty(2 * capacity + capacity // 2, dtype=torch.int32, device=dev).split((capacity, capacity, capacity // 2))
            status = self._sticky_status(dev)
            self._run("radius_graph_capacity", self.lib.mlcgb_graph_capacity,
                      (_ptr(pos), dt, _ptr(n_atoms), _ptr(ptr), N, B, float(r), int(max_num_neighbors), int(rule), _ptr(ws), wsb, _ptr(offsets), capacity,
                       _ptr(rows[0]), _ptr(rows[1]), _ptr(twin), _ptr(sel), _ptr(pair_of), _ptr(counts), _ptr(status), _stream()), launches=7,
                      nbytes=N * 24 + capacity * 8)
        self.defer_status(status, "radius graph with a fixed edge capacity")
        return dict(row0=rows[0], row1=rows[1], offsets=offsets, counts=counts, ptr=ptr, twin=twin, sel=sel, pair_of=pair_of)

    def edge_twin(self, row0, row1, offsets, N, fresh_status: bool = False):
        """twin[e] = position of the reversed edge; second value: the status words (bit 2: an edge without its reverse).  By default
        the words are the backend's accumulating ones; ``fresh_status=True`` gives this call its own."""
        _need_cuda(row0)
        E = row0.numel()
        twin = torch.empty(E, dtype=torch.int32, device=row0.device)
        status = torch.zeros(4, dtype=torch.int32, device=row0.device) if fresh_status else self._sticky_status(row0.device)
        with _on(row0.device):
            self._run("edge_twin", self.lib.mlcgb_edge_twin, (_ptr(row0), _ptr(row1), _ptr(offsets), E, N, _ptr(twin), _ptr(status), _stream(),), **self._work("edge_twin", locals()))
        return twin, status

    def pair_plan(self, row0, row1, offsets, N, fresh_status: bool = False):
        """(twin [E], sel [E/2], pair_of [E], status words) of a symmetric, loop-free, centre-sorted list with an even number of
        edges; status bit 2: a missing reverse edge or a loop."""
        _need_cuda(row0)
        E, dev = row0.numel(), row0.device
        out = torch.zeros(2 * E + E // 2, dtype=torch.int32, device=dev)    # (entries no edge claims stay valid indices)
        twin, pair_of, sel = out[:E], out[E:2 * E], out[2 * E:]
        wsb = self.lib.mlcgb_pair_plan_workspace_bytes(N)
        ws = torch.empty(max(wsb, 1), dtype=torch.uint8, device=dev)
        status = torch.zeros(4, dtype=torch.int32, device=dev) if fresh_status else self._sticky_status(dev)
        with _on(dev):
            self._run("pair_plan", self.lib.mlcgb_pair_plan, (_ptr(row0), _ptr(row1), _ptr(offsets), E, N, _ptr(ws), wsb, _ptr(twin), _ptr(sel), _ptr(pair_of),
                                                               _ptr(status), _stream()), launches=5, nbytes=28 * E + 20 * N)
        return twin, sel, pair_of, status

    def list_plan(self, edge_index, offsets, ptr, N):
        """``(row0, row1, twin, sel, pair_of)``, all int32, of a complete, loop-free list (int64 [2, E], E even and not 0) as
        :meth:`radius_graph` returns it with its offsets and the structure boundaries (or None) it was made with.  A list that is none is
        reported through the accumulating status words."""
        _need_cuda(edge_index, offsets, ptr)
        E, dev = edge_index.shape[1], edge_index.device
        with _on(dev):
            pad = -E % 8            # (row1 on a 32-byte boundary)
            r0, _, r1, twin, pair_of, sel = torch.empty(4 * E + pad + E // 2, dtype=torch.int32, device=dev).split((E, pad, E, E, E, E // 2))
            wsb = self.lib.mlcgb_list_plan_workspace_bytes(N)
            ws = torch.empty(wsb, dtype=torch.uint8, device=dev)
            self._run("list_plan", self.lib.mlcgb_list_plan, (
                _ptr(edge_index), _ptr(offsets), _ptr(ptr), 0 if ptr is None else ptr.numel() - 1, E, N, _ptr(ws), wsb, _ptr(r0), _ptr(r1), _ptr(twin), _ptr(sel),
                _ptr(pair_of), _ptr(self._sticky_status(dev)), _stream()), launches=5, nbytes=46 * E + 20 * N)
        return r0, r1, twin, sel, pair_of

    def pair_index(self, sel, twin):
        """pair_of[e] = k for the k-th selected edge and for its reverse."""
        _need_cuda(sel, twin)
        pair_of = torch.empty(twin.numel(), dtype=torch.int32, device=twin.device)
        with _on(twin.device):
            self._run("pair_index", self.lib.mlcgb_pair_index, (_ptr(sel), _ptr(twin), sel.numel(), _ptr(pair_of), _stream(),), nbytes=12 * sel.numel())
        return pair_of

    # ------------------------------------------------------------------ geometry
    def edge_diff(self, pos, row0, row1):
        _need_cuda(pos, row0, row1)
        pos = pos.contiguous()
        E = row0.numel()
        out = torch.empty((E, 3), dtype=pos.dtype, device=pos.device)
        status = torch.zeros(4, dtype=torch.int32, device=pos.device)
        with _on(pos.device):
            self._run("edge_diff", self.lib.mlcgb_edge_diff, (_ptr(pos), _dt(pos), _ptr(row0), _ptr(row1), E, pos.shape[0], _ptr(out), _ptr(status), _stream(),), **self._work("edge_diff", locals()))
        return out

    def _sticky_status(self, dev):
        """One status array per device for kernels whose status is only ever checked lazily (bits accumulate)."""
        st = self._status.get(dev)
        if st is None:
            with lasting():
                st = self._status[dev] = torch.zeros(4, dtype=torch.int32, device=dev)
        return st

    def edge_distance(self, pos, row0, row1):
        _need_cuda(pos, row0, row1)
        pos = pos.contiguous()
        E = row0.numel()
        out = torch.empty(E, dtype=pos.dtype, device=pos.device)
        with _on(pos.device):
            self._run("edge_distance", self.lib.mlcgb_edge_distance,
                      (_ptr(pos), _dt(pos), _ptr(row0), _ptr(row1), E, pos.shape[0], _ptr(out), _ptr(self._sticky_status(pos.device)), _stream()),
                      nbytes=E * (8 + pos.element_size()) + pos.numel() * pos.element_size())
        return out

    def edge_distance_backward(self, pos, g, d, plan):
        _need_cuda(pos, g, d)
        pos, g, d = pos.contiguous(), g.contiguous(), d.contiguous()
        out = torch.empty_like(pos)
        with _on(pos.device):
            self._run("edge_distance_backward", self.lib.mlcgb_edge_distance_backward,
                      (_ptr(pos), _ptr(g), _ptr(d), _dt(pos), _ptr(plan.row0), _ptr(plan.row1), _ptr(plan.ptr_in), _ptr(plan.perm_in),
                       _ptr(plan.ptr_out), _ptr(plan.perm_out), plan.N, plan.E, _ptr(out), _stream()),
                      nbytes=2 * plan.E * (16 + 2 * pos.element_size()) + 2 * pos.numel() * pos.element_size())
        return out

    def node_scatter_diff(self, g, ptr_in, perm_in, ptr_out, perm_out, N):
        _need_cuda(g)
        g = g.contiguous()
        out = torch.empty((N, 3), dtype=g.dtype, device=g.device)
        with _on(g.device):
            self._run("node_scatter_diff", self.lib.mlcgb_node_scatter_diff, (_ptr(g), _dt(g), _ptr(ptr_in), _ptr(perm_in), _ptr(ptr_out), _ptr(perm_out), N,
                                                        g.shape[0], _ptr(out), _stream(),), **self._work("node_scatter_diff", locals()))
        return out

    # ------------------------------------------------------------------ radial basis
    def _spec(self, spec: RbfSpec, dtype, p0=None, p1=None):
        p0, p1 = spec.p0 if p0 is None else p0, spec.p1 if p1 is None else p1
        if p0.dtype != dtype or p1.dtype != dtype or not (p0.is_contiguous() and p1.is_contiguous()):
            p0 = p0.detach().to(dtype).contiguous()
            p1 = p1.detach().to(dtype).reshape(-1).contiguous()
        s = _lib.RbfSpecStruct(spec.kind, spec.num_rbf, spec.cutoff_kind, 0, spec.lower, spec.upper, spec.alpha, p0.data_ptr(), p1.data_ptr())
        return s, (p0, p1)

    def rbf_expand(self, d, spec: RbfSpec, order: int):
        _need_cuda(d, spec.p0, spec.p1)
        d = d.contiguous()
        s, keep = self._spec(spec, d.dtype)
        out = torch.empty((d.numel(), spec.num_rbf), dtype=d.dtype, device=d.device)
        with _on(d.device):
            self._run("rbf_expand", self.lib.mlcgb_rbf_expand, (_ptr(d), _dt(d), d.numel(), ctypes.byref(s), order, _ptr(out), _stream(),), **self._work("rbf_expand", locals()))
        return out

    def rbf_contract(self, d, G, spec: RbfSpec, order: int):
        _need_cuda(d, G, spec.p0, spec.p1)
        d, G = d.contiguous(), G.contiguous()
        s, keep = self._spec(spec, d.dtype)
        out = torch.empty(d.numel(), dtype=d.dtype, device=d.device)
        with _on(d.device):
            self._run("rbf_contract", self.lib.mlcgb_rbf_contract, (_ptr(d), _ptr(G), _dt(d), d.numel(), ctypes.byref(s), order, _ptr(out), _stream(),), **self._work("rbf_contract", locals()))
        return out

    def rbf_param_contract(self, d, G, c, spec: RbfSpec, order: int):
        """``(gp0 [R], gp1 [R] or [1])``: gradients with respect to the two parameter vectors of the basis of
        ``sum_e c[e] sum_k G[e,k] phi_k^(order)(d_e)`` (``c`` may be ``None``)."""
        _need_cuda(d, G, c, spec.p0, spec.p1)
        d, G = d.contiguous(), G.contiguous()
        c = None if c is None else c.contiguous()
        s, keep = self._spec(spec, d.dtype)
        gp0 = torch.empty(spec.num_rbf, dtype=d.dtype, device=d.device)
        gp1 = torch.empty(spec.p1.numel(), dtype=d.dtype, device=d.device)
        nbytes = self.lib.mlcgb_rbf_param_workspace_bytes(d.numel(), spec.num_rbf, _dt(d))
        ws = torch.empty(max(nbytes, 1), dtype=torch.uint8, device=d.device)
        with _on(d.device):
            self._run("rbf_param_contract", self.lib.mlcgb_rbf_param_contract,
                      (_ptr(d), _ptr(G), _ptr(c), _dt(d), d.numel(), ctypes.byref(s), order, _ptr(ws), nbytes, _ptr(gp0), _ptr(gp1), _stream(),),
                      **self._work("rbf_param_contract", locals()))
        return gp0, gp1

    # ------------------------------------------------------------------ CFConv primitives
    def seg_mul_sum(self, a, V, ptr, nbr, eperm, N):
        _need_cuda(a, V, ptr, nbr)
        a, V = a.contiguous(), V.contiguous()
        F = V.shape[1]
        out = torch.empty((N, F), dtype=V.dtype, device=V.device)
        with _on(V.device):
            self._run("seg_mul_sum", self.lib.mlcgb_seg_mul_sum, (_ptr(a), _ptr(V), _dt(V), _ptr(ptr), _ptr(nbr), _ptr(eperm), N, V.shape[0], F, _ptr(out), _stream(),), **self._work("seg_mul_sum", locals()))
        return out

    def edge_mul(self, a, b, ia, ib):
        _need_cuda(a, b, ia, ib)
        a, b = a.contiguous(), b.contiguous()
        E, F = ia.numel(), a.shape[1]
        out = torch.empty((E, F), dtype=a.dtype, device=a.device)
        with _on(a.device):
            self._run("edge_mul", self.lib.mlcgb_edge_mul, (_ptr(a), _ptr(b), _dt(a), _ptr(ia), _ptr(ib), E, F, _ptr(out), _stream(),), **self._work("edge_mul", locals()))
        return out

    def pair_mul(self, a, b, ia, ib):
        """out[p,:] = a[ia[p],:] * b[ib[p],:] + a[ib[p],:] * b[ia[p],:]."""
        _need_cuda(a, b, ia, ib)
        a, b = a.contiguous(), b.contiguous()
        E, F = ia.numel(), a.shape[1]
        out = torch.empty((E, F), dtype=a.dtype, device=a.device)
        with _on(a.device):
            self._run("pair_mul", self.lib.mlcgb_pair_mul, (_ptr(a), _ptr(b), _dt(a), _ptr(ia), _ptr(ib), E, F, _ptr(out), _stream(),), **self._work("edge_mul", locals()))
        return out

    def tanh_grad(self, mode: int, G, g, y):
        """mode 0: ``g * (1 - y**2)``; mode 1: ``-2 * G * g * y`` (elementwise; ``G`` is ignored in mode 0)."""
        _need_cuda(G, g, y)
        g, y = g.contiguous(), y.contiguous()
        G = None if G is None else G.contiguous()
        out = torch.empty_like(y)
        with _on(y.device):
            self._run("tanh_grad", self.lib.mlcgb_tanh_grad, (int(mode), _ptr(G), _ptr(g), _ptr(y), _dt(y), y.numel(), _ptr(out), _stream(),),
                      nbytes=(3 + mode) * y.numel() * y.element_size(), flops=(3 + mode) * y.numel())
        return out

    def row_scale(self, a, c):
        """out[e,:] = a[e,:] * c[e]."""
        _need_cuda(a, c)
        a, c = a.contiguous(), c.contiguous()
        E, F = a.shape
        out = torch.empty_like(a)
        with _on(a.device):
            self._run("row_scale", self.lib.mlcgb_row_scale, (_ptr(a), _ptr(c), _dt(a), E, F, _ptr(out), _stream(),), nbytes=(2 * a.numel() + E) * a.element_size())
        return out

    def row_dot(self, a, b):
        """out[e] = sum_f a[e,f] * b[e,f]."""
        _need_cuda(a, b)
        a, b = a.contiguous(), b.contiguous()
        E, F = a.shape
        out = torch.empty(E, dtype=a.dtype, device=a.device)
        with _on(a.device):
            self._run("row_dot", self.lib.mlcgb_row_dot, (_ptr(a), _ptr(b), _dt(a), E, F, _ptr(out), _stream(),), nbytes=(2 * a.numel() + E) * a.element_size(),
                      flops=2 * a.numel())
        return out

    # ------------------------------------------------------------------ GEMM
    def gemm(self, mode: int, A, B, bias=None):
        """mode 0: A[M,K] B[N,K]^T (+bias); 1: A[M,K] B[K,N]; 2: A[K,M]^T B[K,N]."""
        _need_cuda(A, B, bias)
        A, B = A.contiguous(), B.contiguous()
        if mode == 0:
            (M, K), N = A.shape, B.shape[0]
        elif mode == 1:
            (M, K), N = A.shape, B.shape[1]
        else:
            (K, M), N = A.shape, B.shape[1]
        dt = _dt(A)
        C = torch.empty((M, N), dtype=A.dtype, device=A.device)
        tc_ok = (N <= 128 and K <= 128) if mode != 2 else (M <= 128 and N <= 128)      # what mlcgb_gemm_tc_supported tests
        if self.tensor_core_gemm and dt == 0 and min(M, N, K) > 0 and tc_ok:
            with _on(A.device):
                wsb = self.lib.mlcgb_gemm_tc_workspace_bytes(mode, M, N, K) if mode == 2 else 0
                ws = torch.empty(wsb, dtype=torch.uint8, device=A.device) if wsb else None
                if bias is not None:
                    bias = bias.contiguous()
                status = self._sticky_status(A.device)
                self._run("gemm_tc", self.lib.mlcgb_gemm_tc, (mode, _ptr(A), _ptr(B), _ptr(bias), M, N, K, _ptr(C), _ptr(ws), wsb, _ptr(status), _stream()),
                          launches=2 if wsb else 1, nbytes=(M * K + N * K + M * N) * 4, flops=2 * M * N * K)
                self.defer_status(status, "tensor-core GEMM")
            return C
        with _on(A.device):
            wsb = self.lib.mlcgb_gemm_workspace_bytes(mode, M, N, K, dt)
            ws = torch.empty(wsb, dtype=torch.uint8, device=A.device) if wsb else None
            if bias is not None:
                bias = bias.contiguous()
            self._run("gemm", self.lib.mlcgb_gemm, (mode, _ptr(A), _ptr(B), _ptr(bias), dt, M, N, K, _ptr(C), _ptr(ws), wsb, _stream(),), **self._work("gemm", locals()))
        return C

    def gemm_tn_colsum(self, G, X):
        """(G^T X, column sums of G): weight and bias gradient of a Linear layer in one pass over G (contraction over rows)."""
        _need_cuda(G, X)
        G, X = G.contiguous(), X.contiguous()
        (K, M), N = G.shape, X.shape[1]
        if (self.tensor_core_gemm and G.dtype == torch.float32 and min(M, N, K) > 0 and N % 4 == 0 and X.data_ptr() % 16 == 0
                and self.lib.mlcgb_gemm_tc_supported(2, M, N, K)):
            C = torch.empty((M, N), dtype=G.dtype, device=G.device)
            cs = torch.empty(M, dtype=G.dtype, device=G.device)
            with _on(G.device):
                wsb = self.lib.mlcgb_gemm_tc_workspace_bytes(2, M, N, K)
                ws = torch.empty(wsb, dtype=torch.uint8, device=G.device)
                status = self._sticky_status(G.device)
                self._run("gemm_tc", self.lib.mlcgb_gemm_tc_tn_colsum, (_ptr(G), _ptr(X), K, M, N, _ptr(C), _ptr(cs), _ptr(ws), wsb, _ptr(status), _stream()),
                          launches=3, nbytes=(M * K + N * K + M * N) * 4, flops=2 * M * N * K)
                self.defer_status(status, "tensor-core GEMM")
            return C, cs
        return self.gemm(2, G, X), G.sum(0)

    EPI_NONE, EPI_TANH, EPI_ADD, EPI_TANH_GRAD, EPI_IN_TANH_GRAD_VEC = 0, 1, 2, 3, 4

    def gemm_fused_ok(self, mode: int, A, B) -> bool:
        """Whether :meth:`gemm_fused` takes these operands (float32, widths multiples of four and <= 128)."""
        if not (self.tensor_core_gemm and A.is_cuda and A.dtype == torch.float32 and A.dim() == 2 and B.dim() == 2):
            return False
        M, K = A.shape
        N = B.shape[0] if mode == 0 else B.shape[1]
        return M > 0 and K % 4 == 0 and N % 4 == 0 and N <= 128 and K <= 128

    def gemm_fused(self, mode: int, A, B, bias=None, aux=None, epilogue: int = 0):
        """Row-wise tensor-core GEMM (mode 0: A B^T + bias, mode 1: A B) with the elementwise step that follows it:
        1 tanh, 2 ``+ aux``, 3 ``* (1 - aux**2)``; 4 transforms the input instead: ``A <- aux[None, :] * (1 - A**2)`` with a
        vector ``aux`` over the columns of A."""
        _need_cuda(A, B, bias, aux)
        A, B = A.contiguous(), B.detach().contiguous()
        M, K = A.shape
        N = B.shape[0] if mode == 0 else B.shape[1]
        C = torch.empty((M, N), dtype=A.dtype, device=A.device)
        if bias is not None:
            bias = bias.detach().contiguous()
        if aux is not None:
            aux = aux.contiguous()
        status = self._sticky_status(A.device)
        with _on(A.device):
            self._run("gemm_tc", self.lib.mlcgb_gemm_tc_fused, (mode, _ptr(A), _ptr(B), _ptr(bias), _ptr(aux), int(epilogue), M, N, K, _ptr(C), _ptr(status), _stream()),
                      nbytes=(M * K + N * K + M * N * (2 if aux is not None else 1)) * 4, flops=2 * M * N * K)
        self.defer_status(status, "tensor-core GEMM")
        return C

    def gemm_chain2(self, backward: bool, A, Wa, ba, Wb, bb, aux):
        """Two 128-wide layers in one kernel.  Forward: ``mid = tanh(A Wa^T + ba)``, ``C = aux + mid Wb^T + bb`` -> ``(mid, C)``;
        backward: ``C = ((A Wa) * (1 - aux**2)) Wb`` -> ``(None, C)``."""
        _need_cuda(A, Wa, ba, Wb, bb, aux)
        A, aux = A.contiguous(), aux.contiguous()
        Wa, Wb = Wa.detach().contiguous(), Wb.detach().contiguous()
        ba = None if ba is None else ba.detach().contiguous()
        bb = None if bb is None else bb.detach().contiguous()
        if A.dtype != torch.float32 or A.shape[1] != 128 or tuple(Wa.shape) != (128, 128) or tuple(Wb.shape) != (128, 128) or aux.shape != A.shape:
            raise ValueError("gemm_chain2 takes float32 operands of width 128")
        M = A.shape[0]
        mid = None if backward else torch.empty_like(A)
        C = torch.empty_like(A)
        status = self._sticky_status(A.device)
        with _on(A.device):
            self._run("gemm_tc", self.lib.mlcgb_gemm_tc_chain2, (int(bool(backward)), _ptr(A), _ptr(Wa), _ptr(ba), _ptr(Wb), _ptr(bb), _ptr(aux), M, _ptr(mid), _ptr(C),
                                                                   _ptr(status), _stream()),
                      nbytes=(3 if backward else 4) * M * 128 * 4 + 2 * 128 * 128 * 4, flops=4 * M * 128 * 128)
        self.defer_status(status, "tensor-core GEMM")
        return mid, C

    # ------------------------------------------------------------------ one interaction block per call
    def interaction_ok(self, x, plan, H, F, H2) -> bool:
        """Whether the per-block entry points take this case; with a profiler attached the individual kernels are launched
        instead, so that each is timed on its own."""
        return (self.profiler is None and self.tensor_core_gemm and x.dtype == torch.float32 and x.shape[0] > 0 and F == 128
                and H <= 128 and H2 <= 128 and H % 4 == 0 and H2 % 4 == 0 and plan.half_selection() is not None)

    def interaction_forward(self, x, d, plan, spec: RbfSpec, conv_cut, W1, fA1, fb1, fA2, W2, b2, W3, b3, precision, save_hidden=True):
        """x + lin(tanh(lin2(aggregate(lin1(x), W(d))))) in one library call; returns (x_new, xl, Wp, a, hs) with ``hs`` the
        filter network's hidden layer kept for the backward (None when ``save_hidden`` is off: the backward recomputes it)."""
        N, H = x.shape
        W1, fA1, fb1, fA2, W2, b2, W3, b3 = (t.contiguous() for t in (W1, fA1, fb1, fA2, W2, b2, W3, b3))
        F, H2 = W1.shape[0], W2.shape[0]
        sel, pair_of = plan.half_selection(), plan.pair_index()
        P, dev = sel.numel(), x.device
        s, keep = self._spec(spec, torch.float32)
        new = lambda *shape: torch.empty(shape, dtype=torch.float32, device=dev)
        xl, Wp, agg, a, out = new(N, F), new(P, F), new(N, F), new(N, H2), new(N, H)
        hs = new(self.lib.mlcgb_filter_hidden_bytes(P) // 4) if save_hidden else None
        status = self._sticky_status(dev)
        with _on(dev):
            _lib.check(self.lib.mlcgb_interaction_forward(
                _ptr(x), _ptr(d), _ptr(plan.ptr_out), _ptr(plan.nbr_out), _ptr(sel), _ptr(pair_of), ctypes.byref(s), int(conv_cut[0]),
                float(conv_cut[1]), float(conv_cut[2]), _ptr(W1), _ptr(fA1), _ptr(fb1), _ptr(fA2), _ptr(W2), _ptr(b2), _ptr(W3), _ptr(b3),
                N, plan.E, P, H, F, H2, int(precision), _ptr(xl), _ptr(Wp), _ptr(hs), _ptr(agg), _ptr(a), _ptr(out), _ptr(status), _stream()),
                "interaction_forward")
        self.defer_status(status, "interaction block (forward)")
        return out, xl, Wp, a, hs

    def interaction_backward(self, g, a, Wp, xl, hs, d, plan, spec: RbfSpec, conv_cut, W1, fA1, fb1, fA2, W2, W3, precision, want_gx=True, want_gd=True):
        N, H = g.shape
        W1, fA1, fb1, fA2, W2, W3 = (t.contiguous() for t in (W1, fA1, fb1, fA2, W2, W3))
        F, H2 = W1.shape[0], W2.shape[0]
        sel, pair_of = plan.half_selection(), plan.pair_index()
        P, dev = sel.numel(), g.device
        s, keep = self._spec(spec, torch.float32)
        new = lambda *shape: torch.empty(shape, dtype=torch.float32, device=dev)
        gy, gagg, gxl = new(N, H2), new(N, F), new(N, F)
        gx = new(N, H) if want_gx else None
        gd = new(plan.E) if want_gd else None
        status = self._sticky_status(dev)
        with _on(dev):
            _lib.check(self.lib.mlcgb_interaction_backward(
                _ptr(g), _ptr(a), _ptr(Wp), _ptr(xl), _ptr(hs), _ptr(d), _ptr(plan.ptr_out), _ptr(plan.nbr_out), _ptr(sel), _ptr(pair_of),
                _ptr(plan.perm_in), _ptr(plan.row0), _ptr(plan.row1), ctypes.byref(s), int(conv_cut[0]), float(conv_cut[1]), float(conv_cut[2]),
                _ptr(W1), _ptr(fA1), _ptr(fb1), _ptr(fA2), _ptr(W2), _ptr(W3), N, plan.E, P, H, F, H2, int(precision),
                _ptr(gy), _ptr(gagg), _ptr(gxl), _ptr(gx), _ptr(gd), _ptr(status), _stream()),
                "interaction_backward")
        self.defer_status(status, "interaction block (backward)")
        return gx, gd

    #: :meth:`radius_graph` takes ``n_atoms`` and ``want_plan``
    plans_with_graph = True

    def schnet_eval(self, pos, types, struct_ptr, plan, spec: RbfSpec, conv_cut, weights, precision, want_grad=True, counts=None, forces=False):
        """Energies [B] and d(sum of energies)/d(pos) [N,3] (its negative with ``forces``) of a standard SchNet in one library call.  ``weights`` is what
        :func:`mlcg_b200.nn.schnet.packed_weights` returns: ``(SchnetWeightsStruct, keep-alive objects)``.  ``counts``: the
        device-side (edges, pairs) of a fixed-capacity graph, whose plan is sized by the capacity."""
        _need_cuda(pos, types, struct_ptr, plan.row0)
        wstruct, _keep = weights
        N, dev = pos.shape[0], pos.device
        B = struct_ptr.numel() - 1
        sel, pair_of = plan.half_selection(), plan.pair_index()
        P = sel.numel()
        s, keep = self._spec(spec, torch.float32)
        wsb = self.lib.mlcgb_schnet_eval_workspace_bytes(N, plan.E, P, wstruct.hidden, wstruct.filters, wstruct.conv_out, wstruct.head_width,
                                                         wstruct.num_blocks)
        ws = torch.empty(wsb, dtype=torch.uint8, device=dev)
        energy = torch.empty(B, dtype=torch.float32, device=dev)
        grad = torch.empty((N, 3), dtype=torch.float32, device=dev) if want_grad else None
        status = self._sticky_status(dev)
        with _on(dev):
            _lib.check((self.lib.mlcgb_schnet_energy_forces if forces else self.lib.mlcgb_schnet_eval_counted)(
                _ptr(pos), _ptr(types), _ptr(struct_ptr), N, B, _ptr(plan.row0), _ptr(plan.row1), _ptr(plan.ptr_out), _ptr(sel), _ptr(pair_of),
                _ptr(plan.perm_in), plan.E, P, _ptr(counts), ctypes.byref(s), int(conv_cut[0]), float(conv_cut[1]), float(conv_cut[2]), ctypes.byref(wstruct),
                int(precision), _ptr(ws), wsb, _ptr(energy), _ptr(grad), _ptr(status), _stream()), "schnet_eval")
        self.defer_status(status, "SchNet evaluation")
        return energy, grad

    def schnet_from_positions(self, pos, types, n_atoms, ptr, r, max_num_neighbors, spec: RbfSpec, conv_cut, weights, precision, forces, edges,
                              training=False):
        """Radius graph and :meth:`schnet_eval` in one library call, the lists kept in its workspace: ``(energy [B], gradient or forces
        [N,3], edge count, None)``; None for a list without edges or cut short.  ``n_atoms`` or ``ptr`` (the other None); ``edges``: a
        guess at the edge count that sizes the workspace (too low costs a second call).  ``training``: the forward pass of
        :meth:`schnet_train_forward` (forces), its state as the last value."""
        w, _keep = weights
        dev = pos.device
        s, keep = self._spec(spec, torch.float32)
        pend = self._take_pending(dev)
        status = self._sticky_status(dev)
        with _on(dev):
            code, host, energy, grad, ws, graph_ws = self.native.evaluate(
                pos, types, n_atoms, ptr, r, max_num_neighbors, ctypes.addressof(s), conv_cut[0], conv_cut[1], conv_cut[2], ctypes.addressof(w), precision,
                forces, training, max(int(edges), 0), pend[0][0] if pend else None, status, _stream())
        if code:
            _lib.check(code, "schnet_evaluate")
        if host[1] & STATUS_SIZES:
            status.bitwise_and_(~STATUS_SIZES)
            _raise_for_status(host[1], "radius graph")
        if pend and host[2]:
            self._raise_pending([int(host[2])], pend)
        if host[4] != _lib.EVALUATE_DONE:
            return None
        E = host[0]
        self.defer_status(status, "SchNet force matching" if training else "SchNet evaluation")
        if not training:
            return energy, grad, E, None
        N, B, ref = grad.shape[0], energy.shape[0], ctypes.byref(w)
        at = (ctypes.c_int64 * 8)()
        self.lib.mlcgb_schnet_evaluate_lists(N, B, E, at)
        places = ((0, 0), (4, at[0]) if ptr is None else (5, 0), (3, at[2]), (3, at[3]), (4, at[1]), (3, at[6]), (3, at[5]), (3, at[7]), (3, at[4]), (1, 0), (2, 0))
        ws = ws[:self.lib.mlcgb_schnet_evaluate_workspace_bytes(N, B, E, spec.num_rbf, ref, 1)]          # (saved with the size that its edges ask for, not that of the guess)
        return energy, grad, E, ForceMatchingState(N, B, E, (types, spec.p0, spec.p1, ws, graph_ws, ptr), places, spec, conv_cut, weights)

    def schnet_fixed_ok(self, N, B, weights) -> bool:
        return bool(self.lib.mlcgb_schnet_evaluate_fixed_ok(N, B, ctypes.byref(weights[0])))

    def schnet_fixed(self, pos, types, n_atoms, ptr, r, max_num_neighbors, spec: RbfSpec, conv_cut, weights, precision, forces, rows):
        """:meth:`schnet_from_positions` for batches that :meth:`schnet_fixed_ok` takes without a host read: lists of as many edges as the int32
        ``rows`` [2, capacity] hold (the neighbours go there), more of them are reported by the deferred status check.  ``(energy, gradient or
        forces)``."""
        _need_cuda(pos, types, n_atoms, ptr, rows)
        capacity = rows.shape[1]
        w, _keep = weights
        pos = pos.detach().contiguous()
        N, dev = pos.shape[0], pos.device
        B = ptr.numel() - 1 if n_atoms is None else n_atoms.numel()
        s, keep = self._spec(spec, torch.float32)
        status, lib, ref = self._sticky_status(dev), self.lib, ctypes.byref(w)
        with _on(dev):
            energy = torch.empty(B, dtype=torch.float32, device=dev)
            grad = torch.empty((N, 3), dtype=torch.float32, device=dev)
            size = lib.mlcgb_schnet_evaluate_workspace_bytes
            gb, wsb = size(N, B, -1, 0, ref, 0), size(N, B, capacity, spec.num_rbf, ref, 0)
            graph_ws, ws = torch.empty(gb, dtype=torch.uint8, device=dev), torch.empty(wsb, dtype=torch.uint8, device=dev)
            _lib.check(lib.mlcgb_schnet_evaluate_fixed(
                pos.data_ptr(), types.data_ptr(), _ptr(n_atoms), _ptr(ptr), N, B, r, max_num_neighbors, ctypes.byref(s), conv_cut[0], conv_cut[1], conv_cut[2],
                ref, precision, int(forces), capacity, rows[1].data_ptr(), graph_ws.data_ptr(), gb, ws.data_ptr(), wsb, energy.data_ptr(), grad.data_ptr(), status.data_ptr(),
                _stream()), "schnet_evaluate_fixed")
        self.defer_status(status, "SchNet evaluation with a fixed edge capacity")
        return energy, grad

    # ------------------------------------------------------------------ one force-matching step
    @staticmethod
    def train_ok(setup) -> bool:
        """Whether the calls below take a model: all widths 128 but the output network's, at most ten blocks and 400 bead types."""
        spec, _, (w, _), precision = setup
        return (precision == 0 and w.hidden == 128 and w.filters == 128 and w.conv_out == 128 and w.num_blocks <= 10 and w.num_types <= 400
                and spec.num_rbf <= 128)

    def schnet_train_forward(self, pos, types, struct_ptr, plan, spec: RbfSpec, conv_cut, weights):
        """(energies [B], forces [N,3], state for :meth:`schnet_train_backward`) of a standard SchNet on a given edge plan."""
        _need_cuda(pos, types, struct_ptr, plan.row0)
        wstruct, _keep = weights
        pos = pos.detach().contiguous()
        N, B, dev = pos.shape[0], struct_ptr.numel() - 1, pos.device
        sel, pair_of = plan.half_selection(), plan.pair_index()
        s, keep = self._spec(spec, torch.float32)
        wsb = self.lib.mlcgb_schnet_train_workspace_bytes(0, N, plan.E, sel.numel(), spec.num_rbf, wstruct.head_width, wstruct.num_blocks, wstruct.num_types)
        ws = torch.empty(wsb, dtype=torch.uint8, device=dev)
        energy = torch.empty(B, dtype=torch.float32, device=dev)
        forces = torch.empty((N, 3), dtype=torch.float32, device=dev)
        status = self._sticky_status(dev)
        with _on(dev):
            _lib.check(self.lib.mlcgb_schnet_train_forward(
                _ptr(pos), _ptr(types), _ptr(struct_ptr), N, B, _ptr(plan.row0), _ptr(plan.row1), _ptr(plan.ptr_out), _ptr(sel), _ptr(pair_of),
                _ptr(plan.perm_in), plan.E, sel.numel(), ctypes.byref(s), int(conv_cut[0]), float(conv_cut[1]), float(conv_cut[2]), ctypes.byref(wstruct), 1,
                _ptr(ws), wsb, _ptr(energy), _ptr(forces), _ptr(status), _stream()), "schnet_train_forward")
        self.defer_status(status, "SchNet force matching")
        tensors = (types, struct_ptr, plan.row0, plan.row1, plan.ptr_out, sel, pair_of, ws, plan.perm_in, spec.p0, spec.p1)
        return energy, forces, ForceMatchingState(N, B, plan.E, tensors, tuple((k, 0) for k in range(len(tensors))), spec, conv_cut, weights)

    def schnet_train_backward(self, state, saved, params, gE, gF):
        """Gradients of a loss on the energies and forces of the forward pass that ``state`` came from with respect to the weights, as
        views of one buffer in the order of the packed weights (``None`` for the output network's second bias).  ``saved``, ``params``:
        the buffers of the state and the weights (without the absent ones) as the autograd node's saved tensors hand them back."""
        wstruct, (_, tensors, live, addresses) = state.weights
        if self.native.pointers(list(params)) != addresses:          # (moved by a saved-tensor hook)
            moved = iter([t.contiguous() for t in params])
            weights = [None if t is None else next(moved) for t in tensors]
            wstruct, _keep = weights_struct(wstruct, weights)
        N, B, E, dev = state.N, state.B, state.E, gF.device
        types, struct_ptr, row0, row1, offsets, sel, pair_of, forward_ws = state.addresses(saved)[:8]
        s, keep = self._spec(state.spec, torch.float32, saved[state.places[-2][0]], saved[state.places[-1][0]])
        wsb = self.lib.mlcgb_schnet_train_workspace_bytes(1, N, E, E // 2, state.spec.num_rbf, wstruct.head_width, wstruct.num_blocks, wstruct.num_types)
        ws = torch.empty(wsb, dtype=torch.uint8, device=dev)
        places = _weights_places(state.weights)
        flat = torch.empty(places.total, dtype=torch.float32, device=dev)
        gs, arr = places.struct(wstruct, flat.data_ptr())
        status = self._sticky_status(dev)
        cut = state.conv_cut
        with _on(dev):
            _lib.check(self.lib.mlcgb_schnet_train_backward(
                types, struct_ptr, N, B, row0, row1, offsets, sel, pair_of, E, E // 2, ctypes.byref(s), int(cut[0]), float(cut[1]), float(cut[2]),
                ctypes.byref(wstruct), 1, _ptr(gE), _ptr(gF), forward_ws, ws.data_ptr(), wsb, ctypes.byref(gs), status.data_ptr(), _stream()),
                "schnet_train_backward")
        self.defer_status(status, "SchNet force matching")
        views = iter(self.native.views(flat, live))                  # (behind the launches: the device is busy by now)
        return [None if t is None or k == 4 else next(views) for k, t in enumerate(tensors)]

    # ------------------------------------------------------------------ fused filter network (tensor cores)
    def filter_forward(self, d, spec: RbfSpec, conv_cutoff_kind, conv_lower, conv_upper, A1, b1, A2, precision=0, sel=None, twin=None, save_hidden=False):
        """W[E,F] = (tanh(phi(d) A1^T + b1) A2^T) * C(d); float32, F = 128, R <= 128.
        ``sel`` / ``twin``: compute one row per unordered pair and write it to both edges (symmetric edge lists);
        ``sel`` alone: W has one row per selected edge, in the order of ``sel``.
        Returns ``(W, status)``, or ``(W, status, hidden)`` with ``save_hidden``: the first layer's output kept (in the kernels'
        own order) for :meth:`filter_backward`."""
        _need_cuda(d, A1, b1, A2, spec.p0, spec.p1)
        if d.dtype != torch.float32:
            raise TypeError("filter_forward is a float32 kernel")
        d, A1, b1, A2 = d.contiguous(), A1.detach().contiguous(), b1.detach().contiguous(), A2.detach().contiguous()
        s, keep = self._spec(spec, d.dtype)
        E, F = d.numel(), A2.shape[0]
        rows = E if sel is None else sel.numel()
        W = torch.empty((E if (sel is None or twin is not None) else rows, F), dtype=d.dtype, device=d.device)
        hs = torch.empty(self.lib.mlcgb_filter_hidden_bytes(rows) // 4, dtype=torch.float32, device=d.device) if save_hidden else None
        status = self._sticky_status(d.device)
        with _on(d.device):
            self._run("filter_forward", self.lib.mlcgb_filter_forward,
                      (_ptr(d), rows, _ptr(sel), _ptr(twin), ctypes.byref(s), int(conv_cutoff_kind), float(conv_lower), float(conv_upper), _ptr(A1), _ptr(b1), _ptr(A2), F,
                       int(precision), _ptr(W), _ptr(hs), _ptr(status), _stream()),
                      nbytes=W.shape[0] * 4 * F + 4 * rows + (hs.numel() * 4 if save_hidden else 0), flops=2 * rows * F * (spec.num_rbf + F))
        return (W, status, hs) if save_hidden else (W, status)

    def filter_backward(self, d, spec: RbfSpec, conv_cutoff_kind, conv_lower, conv_upper, A1, b1, A2, row0, row1, xl, gagg, precision=0,
                        sel=None, twin=None, hidden=None):
        """gd[E] = sum_f (xl[row0] * gagg[row1])_f * dW_f/dd.  ``hidden``: what :meth:`filter_forward` kept for the same
        distances, selection and weights (the hidden layer is recomputed without it)."""
        _need_cuda(d, A1, b1, A2, row0, row1, xl, gagg)
        d, A1, b1, A2 = d.contiguous(), A1.detach().contiguous(), b1.detach().contiguous(), A2.detach().contiguous()
        xl, gagg = xl.detach().contiguous(), gagg.detach().contiguous()
        s, keep = self._spec(spec, d.dtype)
        E, F = d.numel(), A2.shape[0]
        rows = E if sel is None else sel.numel()
        gd = torch.empty(E, dtype=d.dtype, device=d.device)
        status = self._sticky_status(d.device)
        with _on(d.device):
            self._run("filter_backward", self.lib.mlcgb_filter_backward,
                      (_ptr(d), rows, _ptr(sel), _ptr(twin), ctypes.byref(s), int(conv_cutoff_kind), float(conv_lower), float(conv_upper), _ptr(A1), _ptr(b1), _ptr(A2), F,
                       int(precision), _ptr(row0), _ptr(row1), _ptr(xl), _ptr(gagg), xl.shape[0], _ptr(hidden), _ptr(gd), _ptr(status), _stream()),
                      nbytes=E * 16 + 2 * xl.numel() * 4 + (hidden.numel() * 4 if hidden is not None else 0), flops=2 * rows * F * 2 * (spec.num_rbf + F))
        return gd, status

    def segment_sum(self, x, ptr):
        _need_cuda(x, ptr)
        x = x.contiguous()
        B = ptr.numel() - 1
        out = torch.empty(B, dtype=x.dtype, device=x.device)
        with _on(x.device):
            self._run("segment_sum", self.lib.mlcgb_segment_sum, (_ptr(x), _dt(x), _ptr(ptr), B, _ptr(out), _stream(),), **self._work("segment_sum", locals()))
        return out

    # ------------------------------------------------------------------ Langevin integrator
    def langevin_first_half(self, x, v, f, masses, beta_mass_ratio, noise, dt, vscale, noisescale):
        """In place on x and v (both contiguous [N,3])."""
        _need_cuda(x, v, f, masses, beta_mass_ratio, noise)
        assert x.is_contiguous() and v.is_contiguous()
        f, noise = f.contiguous(), noise.contiguous()
        with _on(x.device):
            self._run("langevin_first_half", self.lib.mlcgb_langevin_first_half,
                      (_ptr(x), _ptr(v), _ptr(f), _ptr(masses), _ptr(beta_mass_ratio), _ptr(noise), _dt(x), x.shape[0], float(dt), float(vscale),
                       float(noisescale), _stream()), nbytes=6 * x.numel() * x.element_size())

    def langevin_second_half(self, v, f, masses, dt):
        _need_cuda(v, f, masses)
        assert v.is_contiguous()
        f = f.contiguous()
        with _on(v.device):
            self._run("langevin_second_half", self.lib.mlcgb_langevin_second_half, (_ptr(v), _ptr(f), _ptr(masses), _dt(v), v.shape[0], float(dt), _stream()),
                      nbytes=3 * v.numel() * v.element_size())

    # ------------------------------------------------------------------ priors
    def prior_terms(self, kind, pos, mapping, mapping_batch, params, B, want_grad=True):
        """Returns (energy[B], dE/dpos[N,3] | None)."""
        _need_cuda(pos, mapping, mapping_batch, params)
        pos, mapping, mapping_batch, params = pos.detach().contiguous(), mapping.contiguous(), mapping_batch.contiguous(), params.contiguous()
        M, N = mapping.shape[1], pos.shape[0]
        # the kernel accumulates: one zero-filled buffer holds the gradient (first, so that it stays 16-byte aligned) and the energies
        buf = torch.zeros(3 * N + B if want_grad else B, dtype=pos.dtype, device=pos.device)
        grad = buf[:3 * N].view(N, 3) if want_grad else None
        energy = buf[3 * N:] if want_grad else buf
        status = self._sticky_status(pos.device)       # (bit 1: a term with an index out of range was skipped)
        with _on(pos.device):
            self._run("prior_terms", self.lib.mlcgb_prior_terms, (kind, _ptr(pos), _dt(pos), _ptr(mapping), _ptr(mapping_batch), _ptr(params), params.shape[0], M, N, B,
                                                  _ptr(energy), _ptr(grad), _ptr(status), _stream(),), **self._work("prior_terms", locals()))
        return energy, grad


    def prior_list(self, mapping, types, tables, params, n_beads, pairs):
        """``(idx int32 [order, M], params [P, M], symmetric, starts)`` of an index list as the neighbour-list dictionary holds it (int64
        [order, M]).  ``tables``: the parameters by the types of a term's beads, each [types] * order of one float dtype, or None where
        ``params`` are given.  ``pairs`` (order 2): whether the list holds every term's reverse with the same parameters, and then the
        first terms of its runs of equal first bead, where these are at least eight terms long on average (else None)."""
        _need_cuda(mapping, types, params, *(tables or ()))
        mapping, types = mapping.contiguous(), types.contiguous()
        order, M = mapping.shape
        if tables is not None:
            n_beads = min(n_beads, types.numel())        # (a bead without a type is one that does not exist)
        dev, like = mapping.device, params if tables is None else tables[0]
        if tables is None:
            params, P, kinds = params.contiguous(), params.shape[0], 1
        else:
            P, kinds = len(tables), like.shape[0]
        with _on(dev):
            idx = torch.empty((order, M), dtype=torch.int32, device=dev)
            out = params if tables is None else torch.empty((P, M), dtype=like.dtype, device=dev)
            pairs = bool(pairs) and M > 0 and M % 2 == 0
            wsb = self.lib.mlcgb_prior_list_workspace_bytes(M) if pairs else 0
            ws = torch.empty(wsb, dtype=torch.uint8, device=dev) if pairs else None
            host = (ctypes.c_int64 * 3)()
            self._run("prior_list", self.lib.mlcgb_prior_list_make, (
                _ptr(mapping), order, M, _ptr(types), n_beads, kinds, P, None if tables is None else (ctypes.c_void_p * P)(*(t.data_ptr() for t in tables)),
                _dt(like), _ptr(params), _ptr(idx), None if tables is None else _ptr(out), _ptr(ws), wsb, host if pairs else None,
                _ptr(self._sticky_status(dev)), _stream()), nbytes=M * (12 * order + P * like.element_size()))
            starts = None
            if host[1] and M >= 8 * host[0] and M < 2 ** 31:
                starts = torch.empty(host[0], dtype=torch.int64, device=dev)
                self._run("prior_list_starts", self.lib.mlcgb_prior_list_starts, (_ptr(idx), M, _ptr(ws), wsb, _ptr(starts), _stream()))
        # what the status word says of the lists made so far: known to the host (a pair list), or to be read
        self.lists.made += 1
        self.lists.word = int(host[2]) if pairs else None
        return idx, out, bool(host[1]), starts

    def lists_name_missing(self, dev) -> bool:
        """Whether :meth:`prior_list` has met a bead or a type that does not exist since this was asked last (a host read unless the last list
        was a pair list, whose call has waited; not while recording)."""
        if torch.cuda.is_current_stream_capturing():
            return False
        status, word = self._sticky_status(dev), self.lists.word
        if word is None or word & STATUS_NOT_THERE:
            word = int(status[0])
        if word & STATUS_NOT_THERE:
            status[0] = word & ~(STATUS_NOT_THERE | STATUS_BAD_INDEX)
        return bool(word & STATUS_NOT_THERE)

    def pair_slices(self, idx, params, starts, worth):
        """The slices of a pair list (int32 [2, M], runs of equal first bead from ``starts`` on) as ``mlcgb_prior_list`` takes them:
        ``(slices, beads, offsets, params)``; None where the second beads of a slice lie too far apart or ``worth(slots)`` says that
        the padding takes too many (``slots``: those of lanes with a run)."""
        _need_cuda(idx, params, starts)
        idx, params, starts = idx.contiguous(), params.contiguous(), starts.contiguous()
        M, R, dev = idx.shape[1], starts.numel(), idx.device
        n = (R + 31) // 32
        with _on(dev):
            slices = torch.empty((n, 4), dtype=torch.int32, device=dev)
            step0 = torch.empty(n, dtype=torch.int64, device=dev)
            common = (_ptr(idx), _ptr(params), _dt(params), params.shape[0], M, _ptr(starts), R)
            host = (ctypes.c_int64 * 4)()
            self._run("pair_slices", self.lib.mlcgb_pair_slices, common + (0, None, _ptr(slices), None, None, None, _stream()))
            self._run("pair_slices_plan", self.lib.mlcgb_pair_slices_plan, (_ptr(slices), n, R, _ptr(step0), host, _stream()))
            total, unused, low, span = host
            if low < 0 or span >= 2 ** 16 or total >= 2 ** 31 or not worth(4 * (32 * total - unused)):
                return None
            beads = torch.empty((n, 32), dtype=torch.int32, device=dev)
            offsets = torch.empty((total, 32, 4), dtype=torch.uint16, device=dev)
            packed = torch.empty((params.shape[0], total, 32, 4), dtype=params.dtype, device=dev)
            self._run("pair_slices", self.lib.mlcgb_pair_slices, common + (
                total, _ptr(step0), _ptr(slices), _ptr(beads), _ptr(offsets), _ptr(packed), _stream()))
        return slices, beads, offsets, packed

    def prior_eval(self, lists, pos, batch, B, deterministic=True, forces=False, totals=False):
        """Every prior list of a model in one call.  ``lists``: sequence of ``(kind, idx32 [order, M], params [P, M], symmetric,
        None)``, or ``(kind, None, None, True, (slices, beads, offsets, params))`` for a symmetric pair list in slices as
        ``mlcgb_prior_list`` describes them (at most ``_lib.MAX_PRIOR_SEGMENTS``).  Returns ``(energy [n, B], dE/dpos [n, N, 3])``, one row / block
        per list (``forces``: the negative gradient), and with ``totals`` their sums ``(energy [B], gradient [N, 3])`` over the lists.
        ``deterministic``: sums formed as 64-bit fixed-point integers (bit-identical from run to run)."""
        n = len(lists)
        if n == 0 or n > _lib.MAX_PRIOR_SEGMENTS:
            raise ValueError(f"between 1 and {_lib.MAX_PRIOR_SEGMENTS} prior lists per launch")
        _dt(pos)
        dev, prof = pos.device, self.profiler
        if prof is not None:
            terms = [l[4][2].numel() if l[4] is not None else l[1].shape[1] for l in lists]
            moved = sum(m * ((l[4][3] if l[4] is not None else l[2]).shape[0] * pos.element_size() + (2 if l[4] is not None else 4 * l[1].shape[0]))
                        for m, l in zip(terms, lists))
            event = prof.begin("prior_eval", 4, moved + 2 * pos.numel() * pos.element_size(), 40 * sum(terms))
        with _on(dev):
            code, energy, grad = self.native.prior_eval(lists, pos, batch, B, bool(deterministic), bool(forces), bool(totals), self._sticky_status(dev), _stream())
        if code:
            _lib.check(code, "prior_eval")
        if prof is not None:
            prof.end("prior_eval", event)
        return energy, grad


_backend = None


def get_backend():
    global _backend
    if _backend is None:
        _backend = CudaBackend()   # raises ExtensionMissing if the library is absent
    return _backend
