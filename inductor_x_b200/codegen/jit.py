"""Compile-once loader for generated functor modules.

A generated kernel is a small CUDA translation unit that includes the hand-written
templates (``csrc/ixb/gen.cuh``) and defines one functor ``Body`` plus an ``extern "C"``
launcher.  It is compiled with nvcc for sm_100a the first time it is seen, cached on disk
by content hash and called through ctypes.  This replaces ``NPUCachingAutotuner.precompile``
/ ``_precompile_config`` and the launcher closure they build
(``inductor_x/npu_triton_heuristics.py:53-266``), and ``cached_autotune``'s on-disk cache
(``:302-435``).
"""
from __future__ import annotations

import ctypes
import hashlib
import json
import os
import re
import subprocess
import sys
import threading
import time

import torch

from .. import config

_CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "csrc")
_NVCC_FLAGS = ["-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17", "-lineinfo",
               "-Xcompiler", "-fPIC", "-shared", "-Xcudafe", "--diag_suppress=177"]
_lock = threading.Lock()
_loaded: dict = {}


def _native_launcher():
    """``_ixb_host.Launcher`` (``csrc/host_launch.cpp``); raises if the extension is not built."""
    try:
        from .. import _ixb_host
    except ImportError as e:
        raise ImportError(f"{e}: build the launch extension with `make -C {_CSRC}` (or __graft_entry__.build())") from e
    return _ixb_host.Launcher


class GeneratedKernel:
    """Callable handle of one compiled functor module."""

    def __init__(self, key: str, path: str, meta: dict, src: str = ""):
        self.key = key
        self.path = path
        self.meta = dict(meta)
        self.src = src
        self._launches = 0           # those of the general route
        self.shape = None            # launch shape in use, once a measurement picked one
        self.tuning = None           # [(shape, us)] of the last measurement
        # what wrapper code calls: native, falling back to the general route below for whatever
        # is not a plain launch; it reads the configuration's switches on every call
        self.run = _native_launcher()(self._run_general, vars(config))
        tune = self.meta.get("tune")
        self._tune_pending = bool(
            tune and tune.get("candidates") and tune.get("idempotent") and config.autotune
            and tune.get("rows", 0) * tune.get("row_bytes", 0) >= config.autotune_min_bytes)
        self._bind(path)

    @property
    def launches(self) -> int:
        return self._launches + self.run.launches

    def _bind(self, path: str) -> None:
        self.lib = ctypes.CDLL(path)
        self.fn = self.lib.ixb_gen_launch
        self.fn.restype = ctypes.c_int
        self.fn.argtypes = [ctypes.POINTER(ctypes.c_void_p), ctypes.POINTER(ctypes.c_longlong),
                            ctypes.c_void_p]
        self.path = path
        self._arm()

    def _arm(self) -> None:
        """Plain launches go straight to the module; a pending measurement and the bounds report
        of debug builds need the general route on every call."""
        direct = not self._tune_pending and not self.meta.get("bounds")
        self.run.bind(ctypes.cast(self.fn, ctypes.c_void_p).value if direct else 0)

    def _run_general(self, *args, stream=None, status=None):
        if status is not None:       # what a native launch returned: to be worded, not launched again
            self._raise_on_status(status)
        ptrs, ints, keep = [], [], []
        for a in args:
            if isinstance(a, torch.Tensor):
                if not (a.is_cuda or config.dry_run):
                    # a host tensor: its address means nothing on the device.  A single element
                    # (eager mode lets a 0-dim host tensor meet device tensors) is copied over,
                    # ordered on the current stream; anything larger is a caller's mistake.
                    if a.numel() != 1:
                        raise RuntimeError(f"generated kernel {self.meta.get('name', self.key)}: argument of "
                                           f"shape {tuple(a.shape)} lives on {a.device}, not on a CUDA device")
                    a = a.to(torch.device("cuda", torch.cuda.current_device()))
                    keep.append(a)
                ptrs.append(a.data_ptr())
            else:
                ints.append(int(a))
        if config.dry_run:
            return
        if stream is None:
            stream = torch.cuda.current_stream().cuda_stream
        pa = (ctypes.c_void_p * max(len(ptrs), 1))(*ptrs)
        ia = (ctypes.c_longlong * max(len(ints), 1))(*ints)
        if self._tune_pending and not torch.cuda.is_current_stream_capturing():
            self._tune_pending = False
            self._autotune(pa, ia, stream)
            self._arm()
        if config.profile_bandwidth:
            return self._run_profiled(pa, ia, stream, args)
        rc = self.fn(pa, ia, stream)
        self._launches += 1
        if rc != 0:
            self._raise_on_status(rc)
        if self.meta.get("bounds"):
            self._raise_on_bad_index()

    def _raise_on_status(self, rc: int) -> None:
        hint = (" (a run-time reduced extent beyond the capacity the module was compiled for?)"
                if rc == 1 and self.meta.get("family") == "row" else "")
        raise RuntimeError(f"generated kernel {self.meta.get('name', self.key)} failed to launch: cudaError {rc}{hint}")

    def _raise_on_bad_index(self) -> None:
        """Debug builds: read the module's status words (this synchronises) and report an
        out-of-range data-dependent index as eager mode would."""
        status = (ctypes.c_ulonglong * 2)()
        rc = self.lib.ixb_gen_bounds(status)
        if rc != 0:
            raise RuntimeError(f"reading the bounds status failed: cudaError {rc}")
        if status[0]:
            bad = ctypes.c_longlong(status[1]).value
            raise IndexError(f"generated kernel {self.meta.get('name', self.key)}: {status[0]} index value(s) "
                             f"out of range, e.g. {bad}")

    # ---- measured choice of the launch shape ----------------------------------------------
    # Stands where the reference's autotuner benchmarks its tile configurations and caches the
    # best one (inductor_x/npu_triton_heuristics.py:53-266, 302-435).  The candidates are the
    # same body built with other launch-shape macros; each is timed with CUDA events on the
    # caller's own tensors (the kernel writes only its outputs, so repeating it is harmless)
    # and the fastest is kept, in memory and in a small JSON file beside the modules.
    def _autotune(self, pa, ia, stream) -> None:
        tune = self.meta["tune"]
        default = tuple(tune["default"])
        decision = _read_decision(self.key)
        if decision is not None:
            shape = tuple(decision["shape"])
            if shape != default:
                try:
                    self._bind(compile_source(self.src, shape=shape))
                except RuntimeError:
                    return
            self.shape, self.tuning = shape, [tuple(t) for t in decision.get("timings", [])]
            return
        shapes = [default] + [tuple(c) for c in tune["candidates"]][: config.autotune_max_candidates]
        built = compile_variants(self.src, shapes[1:])
        libs = [(default, self.path)] + [(sh, so) for sh, so in built if so is not None]
        results = []
        n = config.autotune_launches
        for shape, so in libs:
            lib = ctypes.CDLL(so)
            fn = lib.ixb_gen_launch
            fn.restype = ctypes.c_int
            fn.argtypes = self.fn.argtypes
            ok = True
            for _ in range(2):
                ok = ok and fn(pa, ia, stream) == 0
            if not ok:
                continue
            # host clock around a device-wide synchronise on both sides: independent of which
            # stream the caller launches on; n back-to-back launches amortise the enqueue cost
            best = float("inf")
            for _ in range(3):
                torch.cuda.synchronize()
                t0 = time.perf_counter()
                for _ in range(n):
                    ok = ok and fn(pa, ia, stream) == 0
                torch.cuda.synchronize()
                best = min(best, (time.perf_counter() - t0) * 1e6 / n)
            if ok:
                results.append((shape, best, so))
        if not results:
            return
        results.sort(key=lambda r: r[1])
        shape, us, so = results[0]
        self.shape = shape
        self.tuning = [(sh, round(t, 2)) for sh, t, _ in results]
        if so != self.path:
            self._bind(so)
        nbytes = 2.0 * tune["rows"] * tune["row_bytes"]
        _write_decision(self.key, dict(shape=list(shape), us=us, gbs=nbytes / us / 1e3,
                                       timings=[[list(sh), t] for sh, t in self.tuning]))
        if config.autotune_verbose:
            print(f"[ixb autotune] {self.key}: " + ", ".join(f"{sh}={t:.1f}us" for sh, t in self.tuning),
                  file=sys.stderr, flush=True)

    def _run_profiled(self, pa, ia, stream, args):
        """ms / GB / GB/s per launch, from the bytes of the tensor arguments
        (inductor_x/npu_triton_heuristics.py:274-299)."""
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        e0.record()
        rc = self.fn(pa, ia, stream)
        e1.record()
        e1.synchronize()
        if rc != 0:
            raise RuntimeError(f"generated kernel failed to launch: cudaError {rc}")
        ms = e0.elapsed_time(e1)
        tensors = [a for a in args if isinstance(a, torch.Tensor)]
        tensors = tensors[:len(tensors) - self.meta.get("workspaces", 0)]     # (the partial sums of column sums)
        gb = sum(a.numel() * a.element_size() for a in tensors) / 1e9
        print(f"{self.meta.get('name', self.key)}: {ms:.3f}ms    {gb:.3f}GB    {gb / (ms / 1e3):.2f}GB/s")


def _decision_path(key: str) -> str:
    return os.path.join(config.cache_dir, f"tune_{key}.json")


def _read_decision(key: str):
    try:
        with open(_decision_path(key)) as f:
            return json.load(f)
    except (OSError, ValueError):
        return None


def _write_decision(key: str, decision: dict) -> None:
    try:
        tmp = f"{_decision_path(key)}.{os.getpid()}.tmp"
        with open(tmp, "w") as f:
            json.dump(decision, f)
        os.replace(tmp, _decision_path(key))
    except OSError:
        pass


_headers_digest = None


def _template_digest() -> bytes:
    """Digest of the template headers a generated module includes: editing a header must
    not resurrect modules compiled against the old one from the on-disk cache."""
    global _headers_digest
    if _headers_digest is None:
        h = hashlib.sha256()
        inc = os.path.join(_CSRC, "ixb")
        for name in sorted(os.listdir(inc)):
            if name.endswith((".cuh", ".h")):
                with open(os.path.join(inc, name), "rb") as f:
                    h.update(name.encode() + b"\0" + f.read())
        _headers_digest = h.digest()
    return _headers_digest


def source_key(src: str) -> str:
    return hashlib.sha256(_template_digest() + src.encode()).hexdigest()[:24]


SHAPE_MACROS = ("IXB_ROW_TEAM", "IXB_ROW_TEAMS", "IXB_ROW_VPT", "IXB_GEN_MIN_CTAS", "IXB_ROW_PF", "IXB_ROW_KREGS")


def compile_source(src: str, verbose: bool = False, shape=None) -> str:
    """Compile ``src`` into the cache directory (if not already there); returns the .so path.
    ``shape`` = (team, teams, vpt, min_ctas, prefetch, register-resident operands) builds a row
    module in another launch shape than the one its source names."""
    key = source_key(src)
    os.makedirs(config.cache_dir, exist_ok=True)
    suffix = "" if shape is None else "_" + "x".join(str(int(v)) for v in shape)
    so = os.path.join(config.cache_dir, f"ixbgen_{key}{suffix}.so")
    if os.path.exists(so):
        return so
    cu = os.path.join(config.cache_dir, f"ixbgen_{key}.cu")
    if not os.path.exists(cu):
        tmp_cu = f"{cu}.{os.getpid()}.{threading.get_ident()}.tmp"
        with open(tmp_cu, "w") as f:
            f.write(src)
        os.replace(tmp_cu, cu)
    tmp = f"{so}.{os.getpid()}.{threading.get_ident()}.tmp"
    t0 = time.time()
    # A row module states how many CTAs per SM its registers are bounded for.  If ptxas had
    # to spill under that bound the module is rebuilt with a looser one.
    defines = []
    m = re.search(r"#define IXB_GEN_MIN_CTAS (\d+)", src)
    n = int(m.group(1)) if m else None
    if shape is not None:
        team, teams, vpt, n, pf, kregs = (int(v) for v in shape)
        defines = [f"-DIXB_ROW_TEAM={team}", f"-DIXB_ROW_TEAMS={teams}", f"-DIXB_ROW_VPT={vpt}", f"-DIXB_ROW_PF={pf}",
                   f"-DIXB_ROW_KREGS={kregs}"]
    bounds = [None]
    if n is not None:
        bounds = [n] + [b for b in (6, 4, 3, 2, 1) if b < n]
    if shape is not None:
        bounds = [n]          # a candidate is built exactly as named; one that spills is dropped
    for bound in bounds:
        extra = [] if bound is None else [f"-DIXB_GEN_MIN_CTAS={bound}"]
        cmd = ["nvcc", *_NVCC_FLAGS, "-Xptxas", "-v", *defines, *extra, *os.environ.get("IXB_NVCC_EXTRA", "").split(),
               "-I", _CSRC, "-o", tmp, cu]
        proc = subprocess.run(cmd, capture_output=True, text=True)
        if proc.returncode != 0:
            raise RuntimeError(f"nvcc failed for generated kernel {cu}:\n{proc.stderr[-4000:]}")
        spills = [int(x) for x in re.findall(r"(\d+) bytes spill stores", proc.stderr)]
        if shape is not None and spills and max(spills) > config.autotune_spill_bytes:
            os.remove(tmp)
            raise RuntimeError(f"launch shape {shape} spills {max(spills)} bytes")
        if bound in (None, 1) or not any(spills):
            break
    os.replace(tmp, so)
    if verbose:
        print(f"compiled {so} in {time.time() - t0:.1f}s")
    return so


def compile_variants(src: str, shapes):
    """Build ``src`` in each launch shape, in parallel; [(shape, path or None)]."""
    from concurrent.futures import ThreadPoolExecutor

    def one(shape):
        try:
            return shape, compile_source(src, shape=shape)
        except RuntimeError:
            return shape, None

    if not shapes:
        return []
    with ThreadPoolExecutor(max_workers=min(len(shapes), config.compile_threads)) as pool:
        return list(pool.map(one, shapes))


def load_kernel(src: str, **meta) -> GeneratedKernel:
    """Entry point named in generated wrapper code."""
    key = source_key(src)
    with _lock:
        k = _loaded.get(key)
        if k is None:
            k = GeneratedKernel(key, compile_source(src), meta, src)
            _loaded[key] = k
            tune = meta.get("tune")
            if config.dry_run and config.prebuild_candidates and tune and tune.get("candidates"):
                # host-only build step: have every launch shape ready for the measurement
                compile_variants(src, [tuple(c) for c in tune["candidates"]][: config.autotune_max_candidates])
    return k
