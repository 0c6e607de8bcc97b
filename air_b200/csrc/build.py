"""Compiles the CUDA sources of this folder for sm_100a into a shared library of C functions, which wants the CUDA runtime and
nothing else and which any program may load, and entry.cpp into an extension module over it, whose functions are the launchers
(entry); what else the library offers is called through ctypes (library).  There is no fallback: without nvcc, or if a source
does not compile, the import fails with the compiler's message.

Both are built at the first call that needs them, into ``_build/`` beside the sources
(or into $AIR_B200_BUILD_DIR, or a per-user temporary folder if the package folder cannot
be written).  A stamp of the sources' contents and the flags decides whether it is rebuilt.
Each translation unit is compiled by its own nvcc process, a few at a time, and a line is
printed for each that starts and ends, so that a first call does not look hung.
"""
from __future__ import annotations

import ctypes
import hashlib
import os
import shutil
import subprocess
import sys
import sysconfig
import tempfile
import time
from concurrent.futures import ThreadPoolExecutor
from importlib import machinery, util

HERE = os.path.dirname(os.path.abspath(__file__))
ARCH_FLAGS = ["-gencode", "arch=compute_100a,code=sm_100a"]
# --use_fast_math is never given: expf, rsqrtf and divisions keep their accurate forms.
NVCC_FLAGS = ["-O3", "-std=c++17", "-lineinfo", "-Xcompiler", "-fPIC", "-Xcompiler", "-fvisibility=hidden",
              "--expt-relaxed-constexpr"]
LIB_NAME = "libair_b200_kernels.so"
ENTRY, ENTRY_MODULE = "entry.cpp", "air_b200_entry"
ENTRY_NAME = ENTRY_MODULE + ".so"

_lib = None
_entry = None


def sources():
    return sorted(f for f in os.listdir(HERE) if f.endswith(".cu"))


def _headers():
    return sorted(f for f in os.listdir(HERE) if f.endswith((".cuh", ".h")))


def _entries() -> str:
    """entries.inc: prototypes of the launchers, and their places in the module's table of methods."""
    from . import ops
    names = {ctypes.c_void_p: "void*", ctypes.c_int: "int", ctypes.c_longlong: "long long", ctypes.c_float: "float"}
    lines = [f'extern "C" int {f}({", ".join(names[t] for t in types)});' for f, types in ops._SIGNATURES.items()]
    return "\n".join(lines + ["#define AIR_ENTRIES \\"] +
                     [f'    {{"{f}", (PyCFunction)(void (*)(void))Entry<{f}>::call, METH_FASTCALL, nullptr}}, \\' for f in ops._SIGNATURES] +
                     ["", ""])


def _entry_flags():
    """How entry.cpp is compiled and linked: against Python's headers and torch's, and the library beside it."""
    import torch
    root = os.path.dirname(torch.__file__)
    compile_flags = ["-O2", "-std=c++17", "-fPIC", "-fvisibility=hidden", "-w", f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}",
                     "-I", sysconfig.get_paths()["include"], "-I", os.path.join(root, "include"),
                     "-I", os.path.join(root, "include", "torch", "csrc", "api", "include")]
    libraries = ["-l:" + LIB_NAME, "-Wl,-rpath,$ORIGIN", "-L" + os.path.join(root, "lib"), "-ltorch_python", "-ltorch_cpu", "-lc10"]
    return compile_flags, libraries, torch.__version__


def _nvcc() -> str:
    for cand in (os.environ.get("NVCC"), shutil.which("nvcc"), "/usr/local/cuda/bin/nvcc"):
        if cand and os.path.exists(cand):
            return cand
    raise RuntimeError("air_b200: nvcc was not found (set NVCC or add it to PATH); the CUDA kernels "
                       "cannot be built and there is no other implementation")


def _stamp() -> str:
    h = hashlib.sha256()
    for f in sources() + _headers():
        with open(os.path.join(HERE, f), "rb") as fh:
            h.update(f.encode() + b"\0" + fh.read())
    with open(os.path.join(HERE, ENTRY), "rb") as fh:
        h.update(fh.read())
    flags, libraries, version = _entry_flags()
    h.update(" ".join(ARCH_FLAGS + NVCC_FLAGS + flags + libraries + [version, sys.version]).encode() + _entries().encode())
    return h.hexdigest()


def _writable(folder: str) -> bool:
    try:
        os.makedirs(folder, exist_ok=True)
        probe = os.path.join(folder, f".probe{os.getpid()}")
        with open(probe, "w"):
            pass
        os.remove(probe)
        return True
    except OSError:
        return False


def build_dir() -> str:
    env = os.environ.get("AIR_B200_BUILD_DIR")
    if env:
        os.makedirs(env, exist_ok=True)
        return env
    local = os.path.join(HERE, "_build")
    if _writable(local):
        return local
    alt = os.path.join(tempfile.gettempdir(), f"air_b200_build_{os.getuid()}")
    os.makedirs(alt, exist_ok=True)
    return alt


def _say(msg: str) -> None:
    print(f"[air_b200 build] {msg}", file=sys.stderr, flush=True)


def build(force: bool = False, verbose: bool = False) -> str:
    """Builds the library and the module over it if their stamp is stale; returns the library's path."""
    out_dir = build_dir()
    lib, module = os.path.join(out_dir, LIB_NAME), os.path.join(out_dir, ENTRY_NAME)
    stamp_file = os.path.join(out_dir, "stamp.txt")
    stamp = _stamp()
    if not force and os.path.exists(lib) and os.path.exists(module) and os.path.exists(stamp_file):
        with open(stamp_file) as f:
            if f.read().strip() == stamp:
                return lib
    nvcc = _nvcc()
    srcs = sources()
    _say(f"compiling {len(srcs)} CUDA sources for sm_100a into {out_dir}")
    t0 = time.time()

    def compile_one(src):
        obj = os.path.join(out_dir, src[:-3] + ".o")
        cmd = [nvcc] + ARCH_FLAGS + NVCC_FLAGS + (["-Xptxas", "-v"] if verbose else []) + \
              ["-I", HERE, "-c", os.path.join(HERE, src), "-o", obj]
        t = time.time()
        _say(f"  nvcc {src} ...")
        p = subprocess.run(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)
        if p.returncode != 0:
            raise RuntimeError(f"air_b200: nvcc failed on {src}:\n{p.stdout}")
        if verbose and p.stdout:
            print(p.stdout, file=sys.stderr)
        _say(f"  nvcc {src} done in {time.time() - t:.1f} s")
        return obj

    flags, libraries, _ = _entry_flags()

    def compile_entry():
        with open(os.path.join(out_dir, "entries.inc"), "w") as f:
            f.write(_entries())
        obj = os.path.join(out_dir, "entry.o")
        t = time.time()
        _say(f"  c++ {ENTRY} ...")
        p = subprocess.run([os.environ.get("CXX", "g++")] + flags + ["-I", out_dir, "-c", os.path.join(HERE, ENTRY), "-o", obj],
                           stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)
        if p.returncode != 0:
            raise RuntimeError(f"air_b200: the C++ compiler failed on {ENTRY}:\n{p.stdout}")
        _say(f"  c++ {ENTRY} done in {time.time() - t:.1f} s")
        return obj

    def link(command, name, to):
        tmp = to + f".tmp{os.getpid()}"
        p = subprocess.run(command + ["-shared", "-o", tmp], stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)
        if p.returncode != 0:
            raise RuntimeError(f"air_b200: linking {name} failed:\n{p.stdout}")
        os.replace(tmp, to)

    with ThreadPoolExecutor(max_workers=min(8, os.cpu_count() or 2)) as pool:
        entry_obj = pool.submit(compile_entry)
        objs = list(pool.map(compile_one, srcs))
    link([nvcc] + ARCH_FLAGS + objs + ["-Xlinker", "-soname=" + LIB_NAME, "-lcudart"], LIB_NAME, lib)
    link([os.environ.get("CXX", "g++"), entry_obj.result(), "-L" + out_dir] + libraries, ENTRY_NAME, module)
    with open(stamp_file, "w") as f:
        f.write(stamp + "\n")
    _say(f"built {LIB_NAME} in {time.time() - t0:.1f} s")
    return lib


def library() -> ctypes.CDLL:
    """The loaded library (built first if needed)."""
    global _lib
    if _lib is None:
        _lib = ctypes.CDLL(build())
    return _lib


def entry():
    """The extension module over the library: a function per launcher (arguments as in ops._SIGNATURES; it returns the error code)."""
    global _entry
    if _entry is None:
        import torch  # noqa: F401  (the module is linked against it)
        path = os.path.join(os.path.dirname(library()._name), ENTRY_NAME)
        loader = machinery.ExtensionFileLoader(ENTRY_MODULE, path)
        spec = util.spec_from_file_location(ENTRY_MODULE, path, loader=loader)
        module = util.module_from_spec(spec)
        loader.exec_module(module)
        _entry = module
    return _entry
