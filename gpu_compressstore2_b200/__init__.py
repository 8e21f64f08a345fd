"""gpu_compressstore2_b200 — B200-native (sm_100a) bitmask stream compaction.

The operation (compress-store): given a payload column ``T[n]`` and an LSB-first packed
``uint32`` mask of ``n`` bits, write the selected elements contiguously and in order and
return how many were selected. The work is done by the hand-written CUDA kernels in
``libcompressstore.so`` (C ABI: ``include/compressstore.h``); this module is the Python
face of that ABI, with PyTorch used only for device memory and streams.

Reference (RememberOfLife/gpu_compressstore2): the per-call compositions bench1..bench10
(src/benchmarks.cuh:153-440) over intermediate_data scratch (src/benchmarks.cuh:53-151);
``IntermediateData`` and the ``bench_*`` helpers below keep that shape.
"""
from __future__ import annotations

import ctypes
from dataclasses import dataclass

from . import _lib
from ._lib import (
    ALGO_1PASS,
    ALGO_3PASS,
    ALGO_AUTO,
    ALGO_NAIVE,
    COUNT_ERROR,
    SERVE_BATCH,
    SERVE_PER_CALL,
    CsConfig,
    CsError,
    check,
)

__all__ = [
    "ALGO_AUTO", "ALGO_1PASS", "ALGO_3PASS", "ALGO_NAIVE", "COUNT_ERROR", "CsError",
    "compressstore", "compressstore_check", "compressstore_host", "compressstore_release", "Workspace", "IntermediateData", "make_config",
    "popc_chunks", "chunk_prefix_sum", "writeout", "gen_payload", "gen_mask_bernoulli",
    "gen_mask_runs", "gen_mask_dense_prefix", "cub_flagged", "tile_elems", "launch_count",
    "mask_words", "lib", "Batch", "Server", "compressstore_pattern", "pattern_count", "gen_mask_pattern",
    "compressstore_if", "predicate", "ServeResult", "SERVE_BATCH", "SERVE_PER_CALL",
    "Timings", "bench_1pass", "bench_auto", "bench_3pass", "bench_naive",
]

lib = _lib.lib  # loads libcompressstore.so on first use, raising ImportError if it was not built


def _torch():
    import torch

    return torch


_current_raw_stream = None  # () -> handle of the current device's current stream, once CUDA is up


def _stream_handle(stream) -> int | None:
    """cudaStream_t of a torch stream, a handle, or (None) the current stream. The current stream is asked
    of torch's binding directly: torch.cuda.current_stream builds a Stream object per call, 3.5 us of
    the 9 us that a short call took; 0.3 us this way."""
    global _current_raw_stream
    if stream is None:
        if _current_raw_stream is None:
            torch = _torch()
            handle = torch.cuda.current_stream().cuda_stream  # initialises CUDA
            raw, device = torch._C._cuda_getCurrentRawStream, torch._C._cuda_getDevice
            _current_raw_stream = lambda: raw(device())  # noqa: E731
            return handle or None
        return _current_raw_stream() or None
    if isinstance(stream, int):
        return stream or None
    return stream.cuda_stream or None


def _ptr(t) -> int | None:
    return None if t is None else t.data_ptr()


def mask_words(n: int) -> int:
    """Number of uint32 mask words for n elements."""
    return (n + 31) // 32


def tile_elems(elem_bytes: int) -> int:
    return int(lib().cs_tile_elems(elem_bytes))


def launch_count() -> int:
    """Kernel launches issued by libcompressstore.so in this process."""
    return int(lib().cs_launch_count())


def make_config(algo: int = ALGO_AUTO, chunk_length: int = 0, grid_dim: int = 0, skip: int = 0,
                timeout_ns: int = 0, selectivity: float = 0.0) -> CsConfig:
    return CsConfig(algo, chunk_length, grid_dim, skip, timeout_ns, selectivity)


def compressstore(d_in, d_mask, d_out, n: int, d_count, *, algo: int = ALGO_AUTO, chunk_length: int = 0,
                  grid_dim: int = 0, skip: int = 0, timeout_ns: int = 0, selectivity: float = 0.0,
                  workspace: "Workspace | None" = None, stream=None) -> None:
    """Compact ``d_in[:n]`` by ``d_mask`` into ``d_out``; ``d_count`` (uint64/int64 CUDA
    tensor, 1 element) receives the selected count. Asynchronous on ``stream``.
    Element width = ``d_in.element_size()``. ``selectivity``: the fraction the caller expects
    selected (0 = unknown); under ALGO_AUTO it picks the tuning table's entry for that
    selectivity bucket."""
    w = d_in.element_size()
    s = _stream_handle(stream)
    if workspace is None and algo == ALGO_AUTO and not (chunk_length or grid_dim or skip or timeout_ns or selectivity):
        st = lib().compressstore(_ptr(d_in), _ptr(d_mask), _ptr(d_out), n, w, _ptr(d_count), s)
    else:
        cfg = make_config(algo, chunk_length, grid_dim, skip, timeout_ns, selectivity)
        if workspace is None:
            st = lib().compressstore_cfg(_ptr(d_in), _ptr(d_mask), _ptr(d_out), n, w, _ptr(d_count),
                                         ctypes.byref(cfg), s)
        else:
            st = lib().compressstore_ex(_ptr(d_in), _ptr(d_mask), _ptr(d_out), n, w, _ptr(d_count),
                                        workspace.ptr, workspace.nbytes, ctypes.byref(cfg), s)
    check(st, "compressstore")


def _host_ptr(a) -> int:
    """Address of a CPU torch tensor or numpy array."""
    if hasattr(a, "data_ptr"):
        if a.is_cuda:
            raise ValueError("compressstore_host takes host buffers")
        return a.data_ptr()
    return a.ctypes.data


def compressstore_host(h_in, h_mask, h_out, n: int, *, algo: int = ALGO_AUTO, chunk_length: int = 0,
                       timeout_ns: int = 0) -> int:
    """Compact a HOST column (CPU torch tensors or numpy arrays; page-locked memory gives
    full copy/compute overlap) through the device; returns the selected count.
    Element width = the payload's element size."""
    w = h_in.element_size() if hasattr(h_in, "element_size") else h_in.dtype.itemsize
    count = ctypes.c_uint64()
    cfg = make_config(algo, chunk_length, 0, 0, timeout_ns)
    check(lib().compressstore_host(_host_ptr(h_in), _host_ptr(h_mask), _host_ptr(h_out), n, w, ctypes.byref(count),
                                   ctypes.byref(cfg)), "compressstore_host")
    return int(count.value)


def compressstore_release(stream=None) -> None:
    """Free the library-owned scratch kept for ``stream`` on the current device (call it
    before destroying a stream that plain calls ran on)."""
    check(lib().compressstore_release(_stream_handle(stream)), "compressstore_release")


def compressstore_check(stream=None) -> None:
    """Synchronise ``stream``; raise if a bounded device wait of the library-owned
    workspace gave up."""
    check(lib().compressstore_check(_stream_handle(stream)), "compressstore_check")


class Workspace:
    """Caller-owned scratch for compressstore_ex (one call at a time, stream-ordered)."""

    def __init__(self, nbytes: int, device=None, stream=None):
        torch = _torch()
        self.nbytes = int(nbytes + 255) // 256 * 256
        self.buf = torch.empty(self.nbytes + 256, dtype=torch.uint8, device=device or "cuda")
        base = self.buf.data_ptr()
        self.ptr = (base + 255) // 256 * 256
        check(lib().cs_workspace_init(self.ptr, self.nbytes, _stream_handle(stream)), "cs_workspace_init")

    @classmethod
    def for_call(cls, n: int, elem_bytes: int, cfg: CsConfig | None = None, device=None, stream=None) -> "Workspace":
        size = lib().compressstore_workspace_size(n, elem_bytes, ctypes.byref(cfg) if cfg else None)
        if size == 0:
            raise CsError(_lib.ERR_INVALID_VALUE, "compressstore_workspace_size")
        return cls(size, device=device, stream=stream)

    def check(self, stream=None) -> None:
        check(lib().cs_workspace_check(self.ptr, _stream_handle(stream)), "cs_workspace_check")


# ---------------------------------------------------------------------------------------
# The three passes as separate calls
# ---------------------------------------------------------------------------------------
def compressstore_pattern(d_in, d_out, n: int, pattern: int, pattern_length: int, d_count, stream=None) -> None:
    """Compact ``d_in[:n]`` by a periodic selection: element i is kept when bit
    ``i % pattern_length`` of ``pattern`` is set (LSB-first). No mask is read."""
    check(lib().compressstore_pattern(_ptr(d_in), _ptr(d_out), n, d_in.element_size(), pattern & 0xFFFFFFFF,
                                      pattern_length, _ptr(d_count), _stream_handle(stream)), "compressstore_pattern")


PRED_OPS = {"<": _lib.PRED_LT, "<=": _lib.PRED_LE, ">": _lib.PRED_GT, ">=": _lib.PRED_GE, "==": _lib.PRED_EQ,
            "!=": _lib.PRED_NE, "between": _lib.PRED_BETWEEN}


def _elem_type(t) -> tuple[int, str]:
    """cs_elem_type and numpy format of a torch dtype."""
    torch = _torch()
    table = {torch.uint8: (_lib.TYPE_U8, "<u1"), torch.int8: (_lib.TYPE_I8, "<i1"), torch.int16: (_lib.TYPE_I16, "<i2"),
             torch.int32: (_lib.TYPE_I32, "<i4"), torch.int64: (_lib.TYPE_I64, "<i8"),
             torch.float32: (_lib.TYPE_F32, "<f4"), torch.float64: (_lib.TYPE_F64, "<f8")}
    for name, code, fmt in (("uint16", _lib.TYPE_U16, "<u2"), ("uint32", _lib.TYPE_U32, "<u4"),
                            ("uint64", _lib.TYPE_U64, "<u8")):
        if hasattr(torch, name):
            table[getattr(torch, name)] = (code, fmt)
    return table[t]


def predicate(op: str, value, value2=None, elem_type: int | None = None, dtype=None) -> "_lib.CsPredicate":
    """A cs_predicate: ``op`` one of <, <=, >, >=, ==, !=, between (value <= x <= value2);
    the element type is ``elem_type`` (cs_elem_type) or follows the torch ``dtype``."""
    import numpy as np

    if elem_type is None:
        elem_type, fmt = _elem_type(dtype)
    else:
        fmt = ["<u1", "<u2", "<u4", "<u8", "<i1", "<i2", "<i4", "<i8", "<f4", "<f8"][elem_type]

    def bits(v) -> int:
        if v is None:
            return 0
        raw = np.array([v], dtype=fmt).tobytes()
        return int.from_bytes(raw + bytes(8 - len(raw)), "little")

    return _lib.CsPredicate(PRED_OPS[op], elem_type, bits(value), bits(value2))


def compressstore_if(d_in, d_out, n: int, pred, d_count, d_mask_out=None, stream=None) -> None:
    """Compact the elements of ``d_in[:n]`` for which ``pred`` (a cs_predicate, see
    ``predicate``) holds, evaluating it on the device; the selection's mask words go to
    ``d_mask_out`` when given."""
    check(lib().compressstore_if(_ptr(d_in), _ptr(d_out), n, ctypes.byref(pred), _ptr(d_mask_out), _ptr(d_count),
                                 _stream_handle(stream)), "compressstore_if")


def pattern_count(n: int, pattern: int, pattern_length: int) -> int:
    """Selected elements of a periodic selection over n elements."""
    pm = pattern & ((1 << pattern_length) - 1)
    return (n // pattern_length) * bin(pm).count("1") + bin(pm & ((1 << (n % pattern_length)) - 1)).count("1")


def popc_chunks(d_mask, n: int, chunk_length: int, d_counts, stream=None) -> None:
    check(lib().cs_popc_chunks(_ptr(d_mask), n, chunk_length, _ptr(d_counts), _stream_handle(stream)), "cs_popc_chunks")


def chunk_prefix_sum(d_counts, chunk_count: int, d_offsets, d_total=None, workspace: Workspace | None = None,
                     stream=None) -> None:
    if workspace is None:
        workspace = Workspace(lib().cs_scan_workspace_size(chunk_count), stream=stream)
    check(lib().cs_chunk_prefix_sum(_ptr(d_counts), chunk_count, _ptr(d_offsets), _ptr(d_total), workspace.ptr,
                                    workspace.nbytes, _stream_handle(stream)), "cs_chunk_prefix_sum")


def writeout(d_in, d_mask, d_out, n: int, d_offsets, d_counts, chunk_length: int, algo: int = ALGO_3PASS,
             stream=None) -> None:
    check(lib().cs_writeout(_ptr(d_in), _ptr(d_mask), _ptr(d_out), n, d_in.element_size(), _ptr(d_offsets),
                            _ptr(d_counts), chunk_length, algo, _stream_handle(stream)), "cs_writeout")


# ---------------------------------------------------------------------------------------
# Seeded generators (device side; the oracle reproduces them bit for bit)
# ---------------------------------------------------------------------------------------
def gen_payload(d_out, n: int, seed: int, float_unit: bool = False, stream=None) -> None:
    check(lib().cs_gen_payload(_ptr(d_out), n, d_out.element_size(), seed, int(float_unit), _stream_handle(stream)),
          "cs_gen_payload")


def gen_mask_bernoulli(d_mask, n: int, p: float, seed: int, stream=None) -> None:
    check(lib().cs_gen_mask_bernoulli(_ptr(d_mask), n, p, seed, _stream_handle(stream)), "cs_gen_mask_bernoulli")


def gen_mask_runs(d_mask, n: int, mean_run: float, seed: int, stream=None) -> None:
    ws = Workspace(lib().cs_gen_mask_runs_workspace_size(n), stream=stream)
    check(lib().cs_gen_mask_runs(_ptr(d_mask), n, mean_run, seed, ws.ptr, ws.nbytes, _stream_handle(stream)),
          "cs_gen_mask_runs")
    ws.check(stream)


def gen_mask_pattern(d_mask, n: int, pattern: int, pattern_length: int, stream=None) -> None:
    check(lib().cs_gen_mask_pattern(_ptr(d_mask), n, pattern & 0xFFFFFFFF, pattern_length, _stream_handle(stream)),
          "cs_gen_mask_pattern")


def gen_mask_dense_prefix(d_mask, n: int, frac: float, stream=None) -> None:
    check(lib().cs_gen_mask_dense_prefix(_ptr(d_mask), n, frac, _stream_handle(stream)), "cs_gen_mask_dense_prefix")


# ---------------------------------------------------------------------------------------
# Batched form
# ---------------------------------------------------------------------------------------
class Batch:
    """A plan compacting many columns with one launch per pass (cs_batch_* in the C ABI).

    ``columns`` is a list of ``(d_in, d_mask, d_out, n, d_count)`` with CUDA tensors;
    ``d_count`` is a 1-element int64/uint64 tensor (or a view into a larger one). Element
    width = ``d_in.element_size()``. Tensors must outlive the plan (addresses are baked in).
    """

    def __init__(self, columns, timeout_ns: int = 0, stream=None, algo: int = ALGO_AUTO):
        self._keep = list(columns)
        arr = (_lib.CsColumn * max(len(columns), 1))()
        for i, (d_in, d_mask, d_out, n, d_count) in enumerate(columns):
            arr[i] = _lib.CsColumn(_ptr(d_in), _ptr(d_mask), _ptr(d_out), n, d_in.element_size(), 0, _ptr(d_count))
        h = ctypes.c_void_p()
        cfg = make_config(algo=algo, timeout_ns=timeout_ns)
        check(lib().cs_batch_create(ctypes.byref(h), arr, len(columns), ctypes.byref(cfg), _stream_handle(stream)),
              "cs_batch_create")
        self.handle = h

    def run(self, stream=None) -> None:
        check(lib().cs_batch_run(self.handle, _stream_handle(stream)), "cs_batch_run")

    def capture_graph(self, stream=None) -> None:
        check(lib().cs_batch_graph(self.handle, _stream_handle(stream)), "cs_batch_graph")

    def run_per_call(self, stream=None) -> None:
        """The per-call baseline: one plain compressstore per column (a C-side loop)."""
        check(lib().cs_batch_run_per_call(self.handle, _stream_handle(stream)), "cs_batch_run_per_call")

    @property
    def one_pass_columns(self) -> int:
        return int(lib().cs_batch_one_pass_columns(self.handle))

    def check(self, stream=None) -> None:
        check(lib().cs_batch_check(self.handle, _stream_handle(stream)), "cs_batch_check")

    @property
    def device_bytes(self) -> int:
        return int(lib().cs_batch_device_bytes(self.handle))

    @property
    def launches_per_run(self) -> int:
        return int(lib().cs_batch_launches(self.handle))

    def close(self) -> None:
        if getattr(self, "handle", None):
            lib().cs_batch_destroy(self.handle)
            self.handle = None

    def __del__(self):
        try:
            self.close()
        except Exception:  # noqa: BLE001
            pass


# ---------------------------------------------------------------------------------------
# Serving loop (cs_server_* in the C ABI)
# ---------------------------------------------------------------------------------------
@dataclass
class ServeResult:
    """Outcome of one served request (cs_result)."""

    d_out: int | None
    count: int
    latency_ns: int
    queue_ns: int
    status: int
    batch_size: int

    @classmethod
    def of(cls, r) -> "ServeResult":
        return cls(r.d_out, int(r.count), int(r.latency_ns), int(r.queue_ns), int(r.status), int(r.batch_size))


class _DeviceView:
    """Zero-copy view of server-owned device memory for torch.as_tensor."""

    _TYPESTR = {1: "|i1", 2: "<i2", 4: "<i4", 8: "<i8"}

    def __init__(self, ptr: int, count: int, elem_bytes: int):
        self.__cuda_array_interface__ = {"shape": (count,), "typestr": self._TYPESTR[elem_bytes],
                                         "data": (ptr or 0, False), "strides": None, "version": 2}


class Server:
    """Compaction requests over device-resident columns, admitted by an output-memory
    budget and batched as they arrive (cs_server_* in the C ABI).

    ``submit`` takes CUDA tensors (or raw device pointers with ``elem_bytes``) already in
    device memory and returns a ticket; ``wait``/``poll``/``next`` return a
    :class:`ServeResult` whose ``d_out`` lies in the server's arena until ``release``.
    """

    def __init__(self, out_budget_bytes: int = 0, max_batch_elems: int = 0, max_batch: int = 0, slots: int = 0,
                 mode: int = SERVE_BATCH, timeout_ns: int = 0):
        cfg = _lib.CsServerConfig(out_budget_bytes, max_batch_elems, max_batch, slots, mode, 0, timeout_ns)
        h = ctypes.c_void_p()
        check(lib().cs_server_create(ctypes.byref(h), ctypes.byref(cfg)), "cs_server_create")
        self.handle = h
        self._elem_bytes: dict[int, int] = {}

    @staticmethod
    def request(d_in, d_mask, n: int, elem_bytes: int | None = None) -> "_lib.CsRequest":
        if elem_bytes is None:
            elem_bytes = d_in.element_size()
        pin = d_in if isinstance(d_in, int) else _ptr(d_in)
        pm = d_mask if isinstance(d_mask, int) else _ptr(d_mask)
        return _lib.CsRequest(pin, pm, n, elem_bytes, 0)

    def submit(self, d_in, d_mask, n: int, elem_bytes: int | None = None) -> int:
        req = self.request(d_in, d_mask, n, elem_bytes)
        t = ctypes.c_uint64()
        check(lib().cs_server_submit(self.handle, ctypes.byref(req), ctypes.byref(t)), "cs_server_submit")
        self._elem_bytes[t.value] = req.elem_bytes
        return t.value

    def poll(self, ticket: int) -> ServeResult | None:
        r = _lib.CsResult()
        st = lib().cs_server_poll(self.handle, ticket, ctypes.byref(r))
        if st == _lib.PENDING:
            return None
        check(st, "cs_server_poll")
        return ServeResult.of(r)

    def wait(self, ticket: int, timeout_s: float = 0.0) -> ServeResult:
        r = _lib.CsResult()
        st = lib().cs_server_wait(self.handle, ticket, int(timeout_s * 1e9), ctypes.byref(r))
        if st == _lib.PENDING:
            raise TimeoutError(f"request {ticket} not completed within {timeout_s} s")
        check(st, "cs_server_wait")
        return ServeResult.of(r)

    def next(self, timeout_s: float = 0.0) -> tuple[int, ServeResult] | None:
        r = _lib.CsResult()
        t = ctypes.c_uint64()
        st = lib().cs_server_next(self.handle, int(timeout_s * 1e9), ctypes.byref(t), ctypes.byref(r))
        if st == _lib.PENDING:
            return None
        check(st, "cs_server_next")
        return t.value, ServeResult.of(r)

    def output(self, ticket: int, res: ServeResult):
        """The selected elements as a signed-integer tensor VIEW (int8/16/32/64 by width, the
        payload's bits) of the arena; valid until release."""
        torch = _torch()
        w = self._elem_bytes[ticket]
        if res.count == 0:
            dt = {1: torch.int8, 2: torch.int16, 4: torch.int32, 8: torch.int64}[w]
            return torch.empty(0, dtype=dt, device="cuda")
        return torch.as_tensor(_DeviceView(res.d_out, res.count, w), device="cuda")

    def release(self, ticket: int) -> None:
        check(lib().cs_server_release(self.handle, ticket), "cs_server_release")
        self._elem_bytes.pop(ticket, None)

    def stats(self) -> dict:
        st = _lib.CsServerStats()
        check(lib().cs_server_stats_get(self.handle, ctypes.byref(st)), "cs_server_stats_get")
        return {name: int(getattr(st, name)) for name, _ in _lib.CsServerStats._fields_}

    def replay(self, requests, arrival_ns) -> list[ServeResult]:
        """Submit ``requests`` (CsRequest list) at ``arrival_ns`` offsets from now, release
        each completion as it comes; returns one ServeResult per request (d_out None)."""
        n = len(requests)
        reqs = (_lib.CsRequest * max(n, 1))(*requests)
        arr = (ctypes.c_uint64 * max(n, 1))(*[int(a) for a in arrival_ns])
        res = (_lib.CsResult * max(n, 1))()
        check(lib().cs_server_replay(self.handle, reqs, arr, n, res), "cs_server_replay")
        return [ServeResult.of(res[i]) for i in range(n)]

    def close(self) -> None:
        if getattr(self, "handle", None):
            lib().cs_server_destroy(self.handle)
            self.handle = None

    def __enter__(self):
        return self

    def __exit__(self, *exc):
        self.close()

    def __del__(self):
        try:
            self.close()
        except Exception:  # noqa: BLE001
            pass


# ---------------------------------------------------------------------------------------
# CUB DeviceSelect::Flagged comparator (not the product path)
# ---------------------------------------------------------------------------------------
class CubFlagged:
    def __init__(self, n: int, elem_bytes: int, device=None):
        torch = _torch()
        self.temp_bytes = int(_lib.cub().cs_cub_flagged_temp_bytes(n, elem_bytes))
        self.temp = torch.empty(max(self.temp_bytes, 1), dtype=torch.uint8, device=device or "cuda")

    def __call__(self, d_in, d_mask, d_out, n: int, d_count, stream=None) -> None:
        st = _lib.cub().cs_cub_flagged(_ptr(d_in), _ptr(d_mask), _ptr(d_out), n, d_in.element_size(), _ptr(d_count),
                                       _ptr(self.temp), self.temp_bytes, _stream_handle(stream))
        if st != 0:
            raise CsError(st, "cs_cub_flagged")


def cub_flagged(d_in, d_mask, d_out, n: int, d_count, stream=None) -> None:
    CubFlagged(n, d_in.element_size())(d_in, d_mask, d_out, n, d_count, stream)


# ---------------------------------------------------------------------------------------
# Mirror of the reference's operator API shape (src/benchmarks.cuh:53-440)
# ---------------------------------------------------------------------------------------
@dataclass
class Timings:
    """Per-phase milliseconds; -1 = phase not run (src/benchmarks.cuh:10-47)."""

    popc: float = -1.0
    pss1: float = -1.0
    pss2: float = -1.0
    proc: float = -1.0
    total: float = -1.0


class IntermediateData:
    """Scratch owner, the counterpart of intermediate_data (src/benchmarks.cuh:53-151):
    sized once for the largest element count and smallest chunk length, reused per call.
    Holds the plain call's workspace and the buffers of the three separate passes (chunk
    counts, chunk offsets, scan workspace) that the phase-timed compositions use."""

    def __init__(self, element_count: int, chunk_length_min: int, elem_bytes: int, device=None):
        torch = _torch()
        dev = device or "cuda"
        cfg = make_config(ALGO_3PASS, chunk_length_min)
        self.element_count = element_count
        self.chunk_length_min = chunk_length_min
        self.elem_bytes = elem_bytes
        self.ws = Workspace.for_call(element_count, elem_bytes, cfg, device=device)
        chunks = max(1, (element_count + chunk_length_min - 1) // chunk_length_min)
        self.d_counts = torch.zeros(chunks, dtype=torch.int32, device=dev)
        self.d_offsets = torch.zeros(chunks, dtype=torch.int64, device=dev)
        self.scan_ws = Workspace(lib().cs_scan_workspace_size(chunks), device=device)
        self.d_count = torch.zeros(1, dtype=torch.int64, device=dev)
        self.events = [torch.cuda.Event(enable_timing=True) for _ in range(4)]

    def _check_sizes(self, element_count: int, chunk_length: int) -> None:
        if element_count > self.element_count or chunk_length < self.chunk_length_min:
            raise CsError(_lib.ERR_WORKSPACE, "sizes exceed the intermediate data")

    def _run(self, algo: int, d_input, d_mask, d_output, element_count: int, chunk_length: int, grid_size: int) -> Timings:
        """One plain call (the library's fused composition) timed as a whole."""
        self._check_sizes(element_count, chunk_length)
        t = Timings()
        torch = _torch()
        e0, e1 = self.events[0], self.events[3]
        torch.cuda.current_stream().synchronize()
        e0.record()
        compressstore(d_input, d_mask, d_output, element_count, self.d_count, algo=algo, chunk_length=chunk_length,
                      grid_dim=grid_size, workspace=self.ws)
        e1.record()
        e1.synchronize()
        t.total = e0.elapsed_time(e1)
        if algo == ALGO_1PASS:
            t.proc = t.total  # a single kernel: the whole call is the writeout
        return t

    def _run_phases(self, writeout_algo: int, d_input, d_mask, d_output, element_count: int,
                    chunk_length: int) -> Timings:
        """The three passes as separate calls, each timed with CUDA events like the
        reference's compositions time theirs: popc = chunk popcount, pss1 = chunk prefix sum
        (the count lands in d_count), proc = writeout, total = first to last event."""
        self._check_sizes(element_count, chunk_length)
        torch = _torch()
        t = Timings()
        chunks = (element_count + chunk_length - 1) // chunk_length
        counts, offsets = self.d_counts[:max(chunks, 1)], self.d_offsets[:max(chunks, 1)]
        e0, e1, e2, e3 = self.events
        torch.cuda.current_stream().synchronize()
        e0.record()
        popc_chunks(d_mask, element_count, chunk_length, counts)
        e1.record()
        chunk_prefix_sum(counts, chunks, offsets, self.d_count, workspace=self.scan_ws)
        e2.record()
        writeout(d_input, d_mask, d_output, element_count, offsets, counts, chunk_length, writeout_algo)
        e3.record()
        e3.synchronize()
        t.popc = e0.elapsed_time(e1)
        t.pss1 = e1.elapsed_time(e2)
        t.proc = e2.elapsed_time(e3)
        t.total = e0.elapsed_time(e3)
        return t


def bench_1pass(id: IntermediateData, d_input, d_mask, d_output, element_count: int, chunk_length: int = 1024,
                grid_size: int = 0) -> Timings:
    """Single-pass decoupled look-back compaction, timed (no reference counterpart; the
    reference's best composition is bench10, src/benchmarks.cuh:418-440). One kernel, so
    proc = total."""
    return id._run(ALGO_1PASS, d_input, d_mask, d_output, element_count, chunk_length, grid_size)


def bench_auto(id: IntermediateData, d_input, d_mask, d_output, element_count: int, chunk_length: int = 1024,
               grid_size: int = 0) -> Timings:
    """The library's plain call as it runs in production (the tuned form: reduce-then-scan
    pass 1+2 and the writeout, or the 1-pass kernel), timed as a whole."""
    return id._run(ALGO_AUTO, d_input, d_mask, d_output, element_count, chunk_length, grid_size)


def bench_3pass(id: IntermediateData, d_input, d_mask, d_output, element_count: int, chunk_length: int = 1024,
                grid_size: int = 0) -> Timings:
    """popcount -> chunk prefix sum -> writeout as three separate calls with
    per-phase times; the counterpart of bench10 (src/benchmarks.cuh:418-440). grid_size is
    accepted for the reference's signature; the writeout's persistent grid is fixed."""
    return id._run_phases(ALGO_3PASS, d_input, d_mask, d_output, element_count, chunk_length)


def bench_naive(id: IntermediateData, d_input, d_mask, d_output, element_count: int, chunk_length: int = 1024,
                grid_size: int = 0) -> Timings:
    """popcount -> prefix sum -> warp-per-word writeout as three separate calls with
    per-phase times; the counterpart of bench4/bench7 (src/benchmarks.cuh:295-316,360-382)."""
    return id._run_phases(ALGO_NAIVE, d_input, d_mask, d_output, element_count, chunk_length)
