"""Builds the sm_100a kernel library with nvcc and loads it.

Every .cu file of this folder is compiled to an object (`-gencode
arch=compute_100a,code=sm_100a`) and the objects are linked into one shared
library; host_call.cpp becomes the extension module that calls it, on hosts it is written for
(x86-64 Linux with g++ and Python.h; on others ctypes calls it, more slowly).  Both live in
`_build/` beside the sources when that folder can be written, else in a per-user folder under
the system's temporary directory.  A stamp of the sources' contents and the flags decides
whether a build is current, so a fresh checkout compiles once, at its first call, and prints a
line per file while it does.
"""
from __future__ import annotations

import ctypes
import hashlib
import importlib.util
import os
import platform
import re
import shutil
import subprocess
import sys
import sysconfig
import tempfile
import time
from concurrent.futures import ThreadPoolExecutor
from pathlib import Path

HERE = Path(__file__).resolve().parent
LIB_NAME = "libinferflux_b200.so"
HOST_NAME = "_ifx_host" + (sysconfig.get_config_var("EXT_SUFFIX") or ".so")
HOST_FLAGS = ["-O2", "-std=c++17", "-fPIC", "-shared"]
NVCC_FLAGS = ["-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17", "-lineinfo",
              "-Xcompiler", "-fPIC", "--expt-relaxed-constexpr"]
LINK_LIBS = ["-lcublas"]


class BuildError(RuntimeError):
    pass


def _say(msg: str) -> None:
    print(f"[inferflux_b200 build] {msg}", file=sys.stderr, flush=True)


def find_nvcc() -> str:
    for cand in (os.environ.get("NVCC"), shutil.which("nvcc"), "/usr/local/cuda/bin/nvcc"):
        if cand and Path(cand).is_file():
            return cand
    raise BuildError("nvcc not found (looked at $NVCC, PATH and /usr/local/cuda/bin): the CUDA kernels "
                     "cannot be built, and there is no other path")


def sources():
    return sorted(HERE.glob("*.cu"))


def _stamp() -> str:
    h = hashlib.sha256()
    for p in sorted(list(HERE.glob("*.cu")) + list(HERE.glob("*.cuh")) + list(HERE.glob("*.h"))):
        h.update(p.name.encode())
        h.update(p.read_bytes())
    h.update(" ".join(NVCC_FLAGS + LINK_LIBS).encode())
    return h.hexdigest()


def _writable(d: Path) -> bool:
    try:
        d.mkdir(parents=True, exist_ok=True)
        probe = d / f".probe_{os.getpid()}"
        probe.write_text("x")
        probe.unlink()
        return True
    except OSError:
        return False


def build_dir() -> Path:
    in_tree = HERE / "_build"
    if _writable(in_tree):
        return in_tree
    d = Path(tempfile.gettempdir()) / f"inferflux_b200_build_{os.getuid()}"
    if _writable(d):
        return d
    raise BuildError(f"neither {in_tree} nor {d} can be written: nowhere to build the kernels")


def _cuda_lib_dirs():
    dirs = []
    for cand in ("/usr/local/cuda/lib64", "/usr/local/cuda/targets/x86_64-linux/lib",
                 "/usr/local/cuda/lib64/stubs"):
        if Path(cand).is_dir():
            dirs.append(cand)
    return dirs


def _compile_one(nvcc: str, src: Path, obj: Path, verbose_ptxas: bool) -> str:
    cmd = [nvcc, *NVCC_FLAGS, "-c", str(src), "-o", str(obj), "-I", str(HERE)]
    if verbose_ptxas:
        cmd += ["-Xptxas", "-v"]
    t0 = time.time()
    proc = subprocess.run(cmd, capture_output=True, text=True)
    if proc.returncode != 0:
        raise BuildError(f"nvcc failed on {src.name}:\n{proc.stdout}\n{proc.stderr}")
    _say(f"compiled {src.name} in {time.time() - t0:.1f}s")
    return proc.stderr


def _no_extension() -> str:
    """Why host_call.cpp cannot be had on this host, or nothing."""
    if platform.machine() not in ("x86_64", "AMD64") or not sys.platform.startswith("linux"):
        return f"it is written for x86-64 Linux, not for {platform.machine()} {sys.platform}"
    if not (os.environ.get("CXX") or shutil.which("g++")):
        return "no g++"
    include = Path(sysconfig.get_paths()["include"])
    return "" if (include / "Python.h").is_file() else f"no Python.h in {include}"


def _host_stamp() -> str:
    """Of the extension alone: interpreters share a folder and the library, and each has an extension of its own."""
    h = hashlib.sha256((HERE / "host_call.cpp").read_bytes())
    h.update(" ".join(HOST_FLAGS).encode())
    return h.hexdigest()


def _host_is_current(out: Path) -> bool:
    stamp_file = out / (HOST_NAME + ".stamp")
    return (out / HOST_NAME).is_file() and stamp_file.is_file() and stamp_file.read_text().strip() == _host_stamp()


def _compile_host(out: Path) -> None:
    """The extension, unless it is there from these sources."""
    if _host_is_current(out):
        return
    why = _no_extension()
    if why:
        _say(f"host_call.cpp is left out ({why}): kernels are called through ctypes, which takes the host some microseconds more a call")
        return
    gxx = os.environ.get("CXX") or shutil.which("g++")
    include = sysconfig.get_paths()["include"]
    tmp = out / (HOST_NAME + f".tmp{os.getpid()}")
    proc = subprocess.run([gxx, *HOST_FLAGS, "-I", include, str(HERE / "host_call.cpp"), "-o", str(tmp)],
                          capture_output=True, text=True)
    if proc.returncode != 0:
        raise BuildError(f"g++ failed on host_call.cpp:\n{proc.stdout}\n{proc.stderr}")
    os.replace(tmp, out / HOST_NAME)
    (out / (HOST_NAME + ".stamp")).write_text(_host_stamp() + "\n")


def build(force: bool = False, verbose_ptxas: bool = False) -> Path:
    """Compile what is stale and return the path of the shared library."""
    out = build_dir()
    lib, stamp_file = out / LIB_NAME, out / "stamp.txt"
    stamp = _stamp()
    if not force and lib.is_file() and stamp_file.is_file() and stamp_file.read_text().strip() == stamp:
        _compile_host(out)                                   # another interpreter may have built the library
        return lib
    nvcc = find_nvcc()
    srcs = sources()
    _say(f"building {len(srcs)} CUDA sources for sm_100a into {out} (first call or sources changed)")
    objs = [out / (s.stem + ".o") for s in srcs]
    logs = []
    with ThreadPoolExecutor(max_workers=min(8, len(srcs), os.cpu_count() or 1)) as pool:
        for log in pool.map(lambda so: _compile_one(nvcc, so[0], so[1], verbose_ptxas), zip(srcs, objs)):
            logs.append(log)
    tmp = out / (LIB_NAME + f".tmp{os.getpid()}")
    cmd = [nvcc, "-shared", "-o", str(tmp), *[str(o) for o in objs]]
    for d in _cuda_lib_dirs():
        cmd += ["-L", d]
    cmd += LINK_LIBS
    proc = subprocess.run(cmd, capture_output=True, text=True)
    if proc.returncode != 0:
        raise BuildError(f"linking {LIB_NAME} failed:\n{proc.stdout}\n{proc.stderr}")
    os.replace(tmp, lib)
    _compile_host(out)
    stamp_file.write_text(stamp + "\n")
    if verbose_ptxas:
        (out / "ptxas.log").write_text("\n".join(logs))
    _say(f"linked {lib}")
    return lib


_LIB = None


def load_library() -> ctypes.CDLL:
    """The kernel library, built if need be.  Raises if it cannot be had: there is
    no fallback."""
    global _LIB
    if _LIB is None:
        import torch  # noqa: F401  (loads the CUDA runtime and cuBLAS the library links against)
        path = build()
        try:
            _LIB = ctypes.CDLL(str(path))
        except OSError as e:
            raise BuildError(f"cannot load {path}: {e}") from e
    return _LIB


_ENTRY = re.compile(r"\b(int|long long)\s+(ifx_\w+)\s*\(([^()]*)\)\s*\{")


def signatures() -> dict:
    """The C entry points as the sources define them: name -> (whether it returns long long, a letter an argument: p pointer or stream,
    i int, l long long, f float; ? a structure's address, which only ctypes passes)."""
    found = {}
    for src in sources():
        for wide, name, arguments in _ENTRY.findall(re.sub(r"//[^\n]*", "", src.read_text())):
            letters = ""
            for a in filter(None, (a.strip() for a in arguments.split(","))):
                kind = re.sub(r"\s*\w+$", "", a).strip()           # without the argument's name
                if kind.endswith("*"):
                    letters += "?" if "Ifx" in kind else "p"
                else:
                    letters += {"int": "i", "unsigned": "i", "long long": "l", "float": "f", "cudaStream_t": "p"}[kind]
            found[name] = (wide != "int", letters)
    return found


class _ThroughCtypes:
    """One entry point, called as the extension's Function is."""
    KINDS = {"p": ctypes.c_void_p, "i": ctypes.c_int, "l": ctypes.c_longlong, "f": ctypes.c_float}

    def __init__(self, fn, tensor_type, letters):
        fn.argtypes = [self.KINDS[c] for c in letters]
        self._fn, self._tensor, self._letters = fn, tensor_type, letters

    def __call__(self, *args):
        if len(args) != len(self._letters):
            raise TypeError(f"{len(args)} arguments instead of {len(self._letters)}")
        try:
            return self._fn(*[a.data_ptr() if c == "p" and isinstance(a, self._tensor) else a for a, c in zip(args, self._letters)])
        except ctypes.ArgumentError as e:
            raise TypeError(str(e)) from e


class HostLibrary:
    """The kernel library's entry points as callables that take tensors, integers, floats and None as they are, in the count and of the
    kinds that the sources say (TypeError otherwise).  `wide`: the names of those that return long long; all others return int.  Names
    that are not listed are ctypes functions."""

    def __init__(self, library, names, wide, known=None):
        import torch
        known = signatures() if known is None else known
        self._ctypes = library
        host = None
        if _host_is_current(build_dir()):
            spec = importlib.util.spec_from_file_location("_ifx_host", build_dir() / HOST_NAME)
            host = importlib.util.module_from_spec(spec)
            spec.loader.exec_module(host)
        for name in (*names, *wide):
            fn = getattr(self._ctypes, name)
            returns_wide, letters = known[name]
            if returns_wide != (name in wide) or "?" in letters:
                raise BuildError(f"{name} is listed with another result than the sources give it, or takes structures")
            fn.restype = ctypes.c_longlong if returns_wide else ctypes.c_int
            setattr(self, name, _ThroughCtypes(fn, torch.Tensor, letters) if host is None else
                    host.Function(ctypes.cast(fn, ctypes.c_void_p).value, returns_wide, torch.Tensor, letters))

    def __getattr__(self, name):
        return getattr(self._ctypes, name)
