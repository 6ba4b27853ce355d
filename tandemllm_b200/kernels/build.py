"""Builds the CUDA libraries for sm_100a with nvcc and loads them with ctypes.

Sources live in `tandemllm_b200/csrc/`; each library is a list of `.cu` files compiled to objects in
parallel and linked into `csrc/_build/lib<name>-<digest>.so`, the digest taken over the sources, the
shared headers and the flags, so an edited source is rebuilt and a built one is found again (the
reference names its builds by a hash of the text too, engine/native_build.py:26-59). A library is
built at its first use, and only the libraries a run asks for are built. While nvcc runs, a line goes
to stderr for every file. There is no fallback: without nvcc and without a built library the load
fails with the reason.

The sources include no torch header, so a file compiles in seconds; tensors cross as raw pointers and
the stream as a handle.
"""

from __future__ import annotations

import ctypes
import fcntl
import hashlib
import importlib.machinery
import importlib.util
import os
import platform
import shutil
import subprocess
import sys
import sysconfig
import tempfile
import threading
import time
from concurrent.futures import ThreadPoolExecutor

from ..settings import SETTINGS

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "csrc")
ARCH_FLAGS = ["-gencode", "arch=compute_100a,code=sm_100a"]
NVCC_FLAGS = ["-std=c++17", "-O3", "-lineinfo", "-Xcompiler", "-fPIC", "--expt-relaxed-constexpr"]

LIBRARIES: dict[str, list[str]] = {
    # every kernel of the 32-bit path, and the plain bfloat16 variants of the same kernels
    "core": ["rows.cu", "rows_pair.cu", "dyt_act.cu", "gemm_simt.cu", "conv.cu", "attention_simt.cu", "attention_split.cu",
             "attention_headmix.cu", "attention_latent.cu", "attention_flex.cu", "ssm.cu", "recurrence.cu", "recurrence_write.cu",
             "layernorm.cu", "post_norm.cu", "moe_route.cu", "sampling.cu", "graphs.cu"],
    # the tcgen05 / TMA kernels of the bfloat16 path; a 32-bit run never builds or loads them
    "tensorcore": ["tc_gemm.cu", "tc_gemm_pair.cu", "attention_mma.cu", "attention_tc.cu", "attention_headmix_mma.cu",
                   "attention_latent_mma.cu", "attention_flex_mma.cu", "head_linear_mma.cu", "gemm_skinny_mma.cu"],
}
HEADERS = ["common.cuh", "route.cuh", "add_rmsnorm.cuh", "recurrence.cuh", "attention_noalloc.h", "tma.cuh"]

_loaded: dict[str, ctypes.CDLL] = {}
_lock = threading.Lock()


class ExtensionError(RuntimeError):
    """The CUDA library is missing and could not be built."""


def say(text: str) -> None:
    print(f"[tandemllm_b200] {text}", file=sys.stderr, flush=True)


def find_nvcc() -> str | None:
    for cand in (SETTINGS.get("NVCC"), shutil.which("nvcc"), "/usr/local/cuda/bin/nvcc"):
        if cand and os.path.isfile(cand) and os.access(cand, os.X_OK):
            return cand
    return None


def build_dir() -> str:
    """`csrc/_build` in the tree; where the tree cannot be written, a per-user folder under the temp dir."""
    want = SETTINGS.get("BUILD_DIR") or os.path.join(CSRC, "_build")
    try:
        os.makedirs(want, exist_ok=True)
        probe = os.path.join(want, f".w{os.getpid()}")
        with open(probe, "w"):
            pass
        os.remove(probe)
        return want
    except OSError:
        alt = os.path.join(tempfile.gettempdir(), f"tandemllm_b200-build-{os.getuid()}")
        os.makedirs(alt, exist_ok=True)
        return alt


def digest(name: str) -> str:
    h = hashlib.sha1()
    h.update(" ".join(ARCH_FLAGS + NVCC_FLAGS).encode())
    for f in HEADERS + LIBRARIES[name]:
        h.update(f.encode())
        with open(os.path.join(CSRC, f), "rb") as fh:
            h.update(fh.read())
    return h.hexdigest()[:12]


def library_path(name: str, folder: str | None = None) -> str:
    return os.path.join(folder or build_dir(), f"lib{name}-{digest(name)}.so")


def _compile(nvcc: str, src: str, obj: str) -> None:
    cmd = [nvcc, *ARCH_FLAGS, *NVCC_FLAGS, "-I", CSRC, "-c", os.path.join(CSRC, src), "-o", obj]
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0:
        raise ExtensionError(f"nvcc failed on {src}:\n{r.stdout}\n{r.stderr}")


def build(name: str, force: bool = False) -> str:
    """Compile library `name` if its file is not there yet; returns the path of the .so."""
    folder = build_dir()
    out = library_path(name, folder)
    if os.path.isfile(out) and not force:
        return out
    nvcc = find_nvcc()
    if nvcc is None:
        raise ExtensionError(
            f"the CUDA library {os.path.basename(out)} is not built and nvcc was not found "
            "(looked at $TANDEMLLM_NVCC, PATH and /usr/local/cuda/bin/nvcc); this engine has no other path")
    with open(os.path.join(folder, f".{name}.lock"), "w") as lock:
        fcntl.flock(lock, fcntl.LOCK_EX)
        try:
            if os.path.isfile(out) and not force:
                return out
            srcs = LIBRARIES[name]
            tag = digest(name)
            t0 = time.time()
            say(f"building {os.path.basename(out)} for sm_100a: {len(srcs)} files with {nvcc}")
            objs = [os.path.join(folder, f"{name}-{tag}-{os.path.splitext(s)[0]}.o") for s in srcs]
            done = [0]

            def one(pair):
                src, obj = pair
                _compile(nvcc, src, obj)
                done[0] += 1
                say(f"  compiled {src} ({done[0]}/{len(srcs)}, {time.time() - t0:.0f} s)")

            with ThreadPoolExecutor(max_workers=min(len(srcs), os.cpu_count() or 4)) as pool:
                list(pool.map(one, zip(srcs, objs)))
            tmp = out + f".tmp{os.getpid()}"
            r = subprocess.run([nvcc, *ARCH_FLAGS, "-shared", "-o", tmp, *objs], capture_output=True, text=True)
            if r.returncode != 0:
                raise ExtensionError(f"linking {out} failed:\n{r.stdout}\n{r.stderr}")
            os.replace(tmp, out)
            for old in os.listdir(folder):          # builds of earlier source texts are of no use any more
                if old.startswith(f"lib{name}-") and old.endswith(".so") and os.path.join(folder, old) != out:
                    try:
                        os.remove(os.path.join(folder, old))
                    except OSError:
                        pass
            for o in objs:
                try:
                    os.remove(o)
                except OSError:
                    pass
            say(f"built {os.path.basename(out)} in {time.time() - t0:.0f} s")
        finally:
            fcntl.flock(lock, fcntl.LOCK_UN)
    return out


def load(name: str) -> ctypes.CDLL:
    """The loaded library `name`, built first if need be."""
    with _lock:
        if name not in _loaded:
            path = build(name)
            try:
                _loaded[name] = ctypes.CDLL(path)
            except OSError as e:
                raise ExtensionError(f"{path} could not be loaded: {e}") from None
        return _loaded[name]


_KINDS = {ctypes.c_void_p: "p", ctypes.c_longlong: "l", ctypes.c_int: "i", ctypes.c_uint: "i", ctypes.c_float: "f"}


def build_fastcall() -> str | None:
    """The extension that calls launchers (csrc/fastcall.c), compiled if its file is not there yet; None where there is no C compiler, no
    Python header or a compiler that fails, or on another platform than the one it is written for (launches then go through ctypes, as
    they are)."""
    include = sysconfig.get_paths()["include"]
    cc = shutil.which("cc") or shutil.which("gcc")
    source = os.path.join(CSRC, "fastcall.c")
    with open(source, "rb") as fh:
        tag = hashlib.sha1(fh.read() + sys.version.encode()).hexdigest()[:12]
    folder = build_dir()
    out = os.path.join(folder, f"fastcall-{tag}.so")
    if os.path.isfile(out):
        return out
    if platform.machine() != "x86_64" or not sys.platform.startswith("linux") or not cc or not os.path.isfile(os.path.join(include, "Python.h")):
        return None
    tmp = out + f".tmp{os.getpid()}"
    try:
        subprocess.run([cc, "-O2", "-shared", "-fPIC", "-I", include, source, "-o", tmp], capture_output=True, text=True, check=True)
        os.replace(tmp, out)
    except (OSError, subprocess.CalledProcessError) as e:
        say(f"{cc} failed on fastcall.c, launches go through ctypes: {e}\n{getattr(e, 'stderr', '')}")
        return None
    return out


def _launcher_type():
    global _launcher
    if _launcher is None:
        path, _launcher = build_fastcall(), False
        if path is not None:
            try:
                loader = importlib.machinery.ExtensionFileLoader("fastcall", path)
                module = importlib.util.module_from_spec(importlib.util.spec_from_file_location("fastcall", path, loader=loader))
                loader.exec_module(module)
                _launcher = module.Launcher
            except (ImportError, OSError) as e:
                say(f"{path} could not be loaded, launches go through ctypes: {e}")
    return _launcher


_launcher = None


class Launchers:
    """A library whose functions with declared parameters that return an int are called through csrc/fastcall.c; everything else is
    the library's own."""

    def __init__(self, library: ctypes.CDLL, names):
        self._library = library
        launcher = _launcher_type()
        for name in names if launcher else ():
            fn = getattr(library, name)
            kinds = "".join(_KINDS.get(t, "?") for t in fn.argtypes or ("?",))
            if "?" not in kinds and kinds.count("f") <= 8 and len(kinds) - kinds.count("f") <= 48 and fn.restype is ctypes.c_int:
                setattr(self, name, launcher(ctypes.cast(fn, ctypes.c_void_p).value, kinds, fn))

    def __getattr__(self, name):
        return getattr(self._library, name)


def build_all() -> list[str]:
    return [build(name) for name in LIBRARIES] + [path for path in (build_fastcall(),) if path]
