"""Compiles the CUDA sources of this folder for sm_100a and loads them.

Each ``name.cu`` becomes ``_build/libsb_name.so`` next to the sources (or, if that
folder cannot be written, under the system temp folder), built by ``nvcc`` the
first time a kernel of that file is needed and again whenever the source, the
shared header or the flags change.  The libraries export plain C entry points
and are loaded with ``ctypes``; none of them links against torch, so a build takes
seconds (``host.cpp``, the host side of a launch, is an extension module and does).  There is no other implementation behind these entry points: if a
library can be neither found nor built, the call fails.
"""

from __future__ import annotations

import ctypes
import hashlib
import importlib.util
import os
import re
import shutil
import subprocess
import sys
import sysconfig
import tempfile
import threading
import time

HERE = os.path.dirname(os.path.abspath(__file__))

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a",
    "-O3", "-std=c++17", "-lineinfo",
    "-Xcompiler", "-fPIC", "-shared",
]

#: every kernel source of the library; ``build_all`` compiles all of them
SOURCES = (
    "elementwise",
    "rope_cache",
    "attention_rowwise",
    "attention_decode",
    "attention_decode_mma",
    "attention_decode_noalloc",
    "attention_prefill",
    "attention_prefill_tc",
    "linear_small",
    "sgemm",
    "gemm_tcgen05",
    "gemm_prompt_tcgen05",
    "dense_chain",
    "sampling",
    "streams",
    "attention_diff",
    "attention_diff_prefill",
    "attention_diff_prefill_tc",
    "residual32",
    "wkv",
    "attention_latent",
    "attention_latent_prompt",
    "latent_heads",
    "moe",
    "depth",
    "attention_sink",
    "attention_sink_tc",
    "short_conv",
    "sink_conv",
    "state_scan",
    "state_scan_prompt",
    "state_step",
)

_lock = threading.Lock()
_loaded: dict = {}
_host = None


class KernelBuildError(RuntimeError):
    pass


def _nvcc() -> str:
    for cand in (os.environ.get("NVCC"), shutil.which("nvcc"), "/usr/local/cuda/bin/nvcc"):
        if cand and os.path.isfile(cand):
            return cand
    raise KernelBuildError(
        "nvcc was not found (looked at $NVCC, PATH and /usr/local/cuda/bin); the CUDA kernels of "
        "starter_b200 cannot be built and there is no other implementation to fall back to"
    )


_dir_lock = threading.Lock()
_dir = None


def _build_dir() -> str:
    global _dir
    with _dir_lock:
        if _dir is not None:
            return _dir
        local = os.path.join(HERE, "_build")
        try:
            os.makedirs(local, exist_ok=True)
            probe = os.path.join(local, f".w{os.getpid()}")
            with open(probe, "w"):
                pass
            os.remove(probe)
            _dir = local
        except OSError:
            _dir = os.path.join(tempfile.gettempdir(), f"starter_b200_build_{os.getuid()}")
            os.makedirs(_dir, exist_ok=True)
        return _dir


def _headers() -> list:
    return sorted(f for f in os.listdir(HERE) if f.endswith((".cuh", ".h")))


def _included_sources(name: str) -> list:
    """Other ``.cu`` files of this folder that ``name.cu`` includes."""
    found = []
    with open(os.path.join(HERE, name + ".cu"), "r", encoding="utf-8") as handle:
        for line in handle:
            line = line.strip()
            if line.startswith("#include \"") and line.endswith(".cu\""):
                found.append(line[len("#include \""):-1])
    return found


def _digest(name: str) -> str:
    h = hashlib.sha256()
    h.update(" ".join(NVCC_FLAGS).encode())
    for fname in [name + ".cu"] + _included_sources(name) + _headers():
        with open(os.path.join(HERE, fname), "rb") as handle:
            h.update(fname.encode())
            h.update(handle.read())
    return h.hexdigest()[:16]


def library_path(name: str) -> str:
    """Path of the built library for ``name.cu``, compiling it first if it is missing or stale."""
    src = os.path.join(HERE, name + ".cu")
    if not os.path.isfile(src):
        raise KernelBuildError(f"no kernel source {src}")
    out_dir = _build_dir()
    lib = os.path.join(out_dir, f"libsb_{name}.so")
    stamp = lib + ".stamp"
    digest = _digest(name)
    if os.path.isfile(lib) and os.path.isfile(stamp):
        with open(stamp) as handle:
            if handle.read().strip() == digest:
                return lib
    tmp = f"{lib}.{os.getpid()}.tmp"
    cmd = [_nvcc()] + NVCC_FLAGS + ["-I", HERE, "-o", tmp, src]
    print(f"[starter_b200] compiling {name}.cu for sm_100a ...", file=sys.stderr, flush=True)
    started = time.monotonic()
    proc = subprocess.Popen(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)
    while True:
        try:
            out, _ = proc.communicate(timeout=15)
            break
        except subprocess.TimeoutExpired:
            print(f"[starter_b200] ... still compiling {name}.cu "
                  f"({time.monotonic() - started:.0f} s)", file=sys.stderr, flush=True)
    if proc.returncode != 0:
        if os.path.exists(tmp):
            os.remove(tmp)
        raise KernelBuildError(f"nvcc failed on {name}.cu:\n{out}")
    os.replace(tmp, lib)
    with open(stamp, "w") as handle:
        handle.write(digest)
    print(f"[starter_b200] built {os.path.basename(lib)} in {time.monotonic() - started:.1f} s",
          file=sys.stderr, flush=True)
    return lib


_ENTRY = re.compile(r"^(int|void|long long)\s+(sb_\w+)\s*\(([^)]*)\)\s*\{", re.M)
_C_TYPES = {"int": ctypes.c_int, "long long": ctypes.c_longlong, "unsigned long long": ctypes.c_ulonglong,
            "float": ctypes.c_float, "cudaStream_t": ctypes.c_void_p}


def declarations(name: str) -> dict:
    """``{entry point: (result type, argument types)}`` of ``name.cu`` as ctypes, read from its source."""
    out = {}
    for fname in [name + ".cu"] + _included_sources(name):
        with open(os.path.join(HERE, fname), "r", encoding="utf-8") as handle:
            for result, entry, params in _ENTRY.findall(handle.read()):
                types = []
                for param in (" ".join(p.split()) for p in params.split(",")):
                    if param in ("", "void"):
                        continue
                    types.append(ctypes.c_void_p if "*" in param else _C_TYPES[param.rsplit(" ", 1)[0]])
                out[entry] = (None if result == "void" else _C_TYPES[result], types)
    return out


def host_path() -> str:
    """Path of the built extension module of ``host.cpp`` (the host side of a launch), compiled first if it is missing or
    stale.  It is the one part that links against torch."""
    import torch

    root = os.path.dirname(torch.__file__)
    compiler = os.environ.get("CXX") or shutil.which("g++") or shutil.which("c++")
    cuda = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(_nvcc()))), "include")
    src = os.path.join(HERE, "host.cpp")
    flags = ["-O2", "-std=c++17", "-fPIC", "-shared", f"-D_GLIBCXX_USE_CXX11_ABI={int(torch.compiled_with_cxx11_abi())}",
             "-I", os.path.join(root, "include"), "-I", os.path.join(root, "include", "torch", "csrc", "api", "include"),
             "-I", cuda, "-I", sysconfig.get_paths()["include"]]
    link = ["-L", os.path.join(root, "lib"), "-ltorch_python", "-ltorch_cuda", "-ltorch_cpu", "-ltorch", "-lc10_cuda", "-lc10",
            "-Wl,-rpath," + os.path.join(root, "lib")]
    lib = os.path.join(_build_dir(), "sb_host.so")
    stamp = lib + ".stamp"
    h = hashlib.sha256(" ".join([torch.__version__, sys.version] + flags + link).encode())
    with open(src, "rb") as handle:
        h.update(handle.read())
    digest = h.hexdigest()[:16]
    if os.path.isfile(lib) and os.path.isfile(stamp):
        with open(stamp) as handle:
            if handle.read().strip() == digest:
                return lib
    if compiler is None:
        raise KernelBuildError("no C++ compiler was found (looked at $CXX and PATH for g++ and c++)")
    tmp = f"{lib}.{os.getpid()}.tmp"
    print("[starter_b200] compiling host.cpp ...", file=sys.stderr, flush=True)
    proc = subprocess.run([compiler] + flags + ["-o", tmp, src] + link, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)
    if proc.returncode != 0:
        if os.path.exists(tmp):
            os.remove(tmp)
        raise KernelBuildError(f"{compiler} failed on host.cpp:\n{proc.stdout}")
    os.replace(tmp, lib)
    with open(stamp, "w") as handle:
        handle.write(digest)
    return lib


def load_host():
    """The extension module of ``host.cpp`` (built on first use)."""
    global _host
    with _lock:
        if _host is None:
            import torch  # noqa: F401  (its libraries have to be there first)

            spec = importlib.util.spec_from_file_location("sb_host", host_path())
            module = importlib.util.module_from_spec(spec)
            spec.loader.exec_module(module)
            _host = module
        return _host


def load(name: str) -> ctypes.CDLL:
    """The loaded library of ``name.cu`` (built on first use).  Its entry points know their argument types, so callers
    pass addresses as plain integers."""
    with _lock:
        lib = _loaded.get(name)
        if lib is None:
            lib = ctypes.CDLL(library_path(name))
            for entry, (result, types) in declarations(name).items():
                function = getattr(lib, entry)
                function.restype, function.argtypes = result, types
            _loaded[name] = lib
        return lib


def build_all(names=SOURCES) -> list:
    """Compile every kernel source and the host module (in parallel) and return the library paths."""
    results = {}
    errors = []

    def work(n):
        try:
            results[n] = host_path() if n == "host" else library_path(n)
        except Exception as exc:  # noqa: BLE001 - collected and re-raised below
            errors.append(exc)

    threads = [threading.Thread(target=work, args=(n,)) for n in list(names) + ["host"]]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    if errors:
        raise errors[0]
    return [results[n] for n in list(names) + ["host"]]
