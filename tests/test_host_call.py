"""Calls of C entry points by host_call.cpp against the same calls through ctypes (no GPU: a small library of its own)."""
import ctypes
import importlib
import importlib.util
import random
import shutil
import subprocess

import pytest
import torch

build = importlib.import_module("inferflux_b200.csrc.build")
# p pointer, i int, l long long, f float; more integers than registers, floats between them, both many
SIGNATURES = ["i", "p", "f", "pilf", "pppppp", "ppppppp", "fiiiiiiiiif", "pppllliiifffpppiiilllfffpp", "l" * 54, "f" * 8 + "p" * 30, "ilp" * 18]


@pytest.fixture(scope="module")
def library(tmp_path_factory):
    if shutil.which("g++") is None:
        pytest.skip("no g++")
    d = tmp_path_factory.mktemp("host_call")
    types = {"p": "const void*", "i": "int", "l": "long long", "f": "float"}
    code = ["#include <stdint.h>"]
    for n, sig in enumerate(SIGNATURES):
        args = ", ".join(f"{types[c]} a{i}" for i, c in enumerate(sig))
        terms = "".join(f" h = h * 1000003 + (long long){'(uintptr_t)' if c == 'p' else ''}a{i}{' * 4096.0f' if c == 'f' else ''};".replace(
            f"(long long)a{i} * 4096.0f", f"(long long)(a{i} * 4096.0f)") for i, c in enumerate(sig))
        code.append(f'extern "C" long long w{n}({args}) {{ unsigned long long h = 1;{terms} return (long long)h; }}')
        code.append(f'extern "C" int n{n}({args}) {{ return (int)w{n}({", ".join(f"a{i}" for i in range(len(sig)))}); }}')
    (d / "f.cpp").write_text("\n".join(code))
    subprocess.run(["g++", "-shared", "-fPIC", "-O1", str(d / "f.cpp"), "-o", str(d / "f.so")], check=True)
    build._compile_host(d)
    spec = importlib.util.spec_from_file_location("_ifx_host", d / build.HOST_NAME)
    host = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(host)
    return ctypes.CDLL(str(d / "f.so")), host


def _arguments(sig, r):
    """(as a program passes them, as ctypes wants them)"""
    plain, wrapped = [], []
    for c in sig:
        if c == "p":
            t = None if r.random() < 0.2 else torch.zeros(3)
            plain.append(t)
            wrapped.append(ctypes.c_void_p(0 if t is None else t.data_ptr()))
        elif c == "f":
            x = r.choice([0.0, -1.5, 0.1, 3e5])
            plain.append(x)
            wrapped.append(ctypes.c_float(x))
        else:
            x = r.choice([0, -1, True, 7, -(1 << 31), (1 << 31) - 1] + ([1 << 40, -(1 << 45)] if c == "l" else []))
            plain.append(x)
            wrapped.append((ctypes.c_int if c == "i" else ctypes.c_longlong)(x))
    return plain, wrapped


@pytest.mark.parametrize("n", range(len(SIGNATURES)))
def test_as_through_ctypes(library, n):
    lib, host = library
    r = random.Random(n)
    for name, kind in ((f"w{n}", ctypes.c_longlong), (f"n{n}", ctypes.c_int)):
        fn = getattr(lib, name)
        fn.restype = kind
        fast = host.Function(ctypes.cast(fn, ctypes.c_void_p).value, kind is ctypes.c_longlong, torch.Tensor)
        for _ in range(20):
            plain, wrapped = _arguments(SIGNATURES[n], r)
            assert fast(*plain) == fn(*wrapped) == fast(*wrapped)


def test_what_it_refuses(library):
    lib, host = library
    fast = host.Function(ctypes.cast(lib.w0, ctypes.c_void_p).value, True, torch.Tensor)
    for args, error in ((("x",), AttributeError), (([1],), AttributeError), ((1.0,) * 9, TypeError), ((1,) * 55, TypeError)):
        with pytest.raises(error):
            fast(*args)
    with pytest.raises(TypeError):
        fast(a=1)


@pytest.mark.parametrize("n", range(len(SIGNATURES)))
def test_a_signature_changes_no_call(library, n):
    lib, host = library
    r = random.Random(100 + n)
    fn = getattr(lib, f"w{n}")
    fn.restype = ctypes.c_longlong
    fast = host.Function(ctypes.cast(fn, ctypes.c_void_p).value, True, torch.Tensor, SIGNATURES[n])
    for _ in range(20):
        plain, wrapped = _arguments(SIGNATURES[n], r)
        assert fast(*plain) == fn(*wrapped) == fast(*wrapped)
        assert fast(*[p.data_ptr() if isinstance(p, torch.Tensor) else p for p in plain]) == fn(*wrapped)


@pytest.mark.parametrize("n", range(len(SIGNATURES)))
def test_another_count_or_kind_is_refused(library, n):
    """What a call without a signature reads from the wrong register, or from whatever lies on the stack."""
    lib, host = library
    r = random.Random(200 + n)
    sig, fn = SIGNATURES[n], getattr(lib, f"w{n}")
    fn.restype = ctypes.c_longlong
    fast = host.Function(ctypes.cast(fn, ctypes.c_void_p).value, True, torch.Tensor, sig)
    plain, wrapped = _arguments(sig, r)
    for wrong in (plain[:-1], plain + [1], plain + [None]):
        with pytest.raises(TypeError):
            fast(*wrong)
    for i, c in enumerate(sig):
        for wrong in {"p": (1.5,), "i": (1.5, None, torch.zeros(1)), "l": (1.5, None, torch.zeros(1)), "f": (None, torch.zeros(1))}[c]:
            with pytest.raises(TypeError):
                fast(*plain[:i], wrong, *plain[i + 1:])
    if "f" in sig:                                           # an integer in the place of a float is one
        whole, as_float = ([7 if c == "f" else p for c, p in zip(sig, plain)], [ctypes.c_float(7.0) if c == "f" else w for c, w in zip(sig, wrapped)])
        assert fast(*whole) == fn(*as_float)


def test_signatures_as_the_sources_have_them():
    known = build.signatures()
    assert known["ifx_embed"] == (False, "pppiiiip") and known["ifx_moe_route_kind"] == (False, "ppppiiiifp")
    assert known["ifx_gemm_f32_split_scratch"] == (True, "iii") and "?" in known["ifx_layer_forward"][1]
    assert sum(letters.count("f") for _wide, letters in known.values()) > 50


@pytest.mark.parametrize("without", ["extension", "python.h", "x86"])
def test_hosts_without_the_extension(library, monkeypatch, tmp_path, capsys, without):
    """Another processor, no g++ or no Python.h: nothing is built and nothing raised, and ctypes makes the same calls and refusals."""
    lib, _ = library
    monkeypatch.setattr(build, "build_dir", lambda: tmp_path)
    if without == "x86":
        monkeypatch.setattr(build.platform, "machine", lambda: "aarch64")
    elif without == "python.h":
        monkeypatch.setattr(build.sysconfig, "get_paths", lambda: {"include": str(tmp_path)})
    else:
        monkeypatch.delenv("CXX", raising=False)
        monkeypatch.setattr(build.shutil, "which", lambda name: None)
    build._compile_host(tmp_path)
    assert not list(tmp_path.iterdir())
    names = [f"n{n}" for n in range(len(SIGNATURES))], [f"w{n}" for n in range(len(SIGNATURES))]
    known = {f"{c}{n}": (c == "w", sig) for c in "nw" for n, sig in enumerate(SIGNATURES)}
    host = build.HostLibrary(ctypes.CDLL(lib._name), *names, known)
    for n, sig in enumerate(SIGNATURES):
        r = random.Random(300 + n)
        for name in (f"n{n}", f"w{n}"):
            plain, wrapped = _arguments(sig, r)
            fn = getattr(lib, name)
            fn.restype = ctypes.c_longlong if name[0] == "w" else ctypes.c_int
            assert getattr(host, name)(*plain) == fn(*wrapped)
            for wrong in (plain[:-1], plain + [1], [1.5 if c != "f" else None for c in sig]):
                with pytest.raises(TypeError):
                    getattr(host, name)(*wrong)


def test_an_extension_of_earlier_sources_is_made_again(monkeypatch, tmp_path):
    """The library's stamp is every interpreter's; each one's extension has its own.  One of earlier sources that cannot be made again is
    not loaded."""
    if shutil.which("g++") is None:
        pytest.skip("no g++")
    import os
    monkeypatch.setattr(build, "build_dir", lambda: tmp_path)
    monkeypatch.setattr(build, "HERE", tmp_path / "sources")
    (tmp_path / "sources").mkdir()
    own = tmp_path / "sources" / "host_call.cpp"
    shutil.copy(os.path.join(os.path.dirname(build.__file__), "host_call.cpp"), own)
    (tmp_path / build.LIB_NAME).write_bytes(b"")
    (tmp_path / "stamp.txt").write_text(build._stamp() + "\n")                # another interpreter has built the library
    host = tmp_path / build.HOST_NAME
    host.write_bytes(b"an extension of earlier sources")
    assert build.build() == tmp_path / build.LIB_NAME
    made = host.stat()
    assert made.st_size > 1000
    build.build()
    assert host.stat().st_mtime_ns == made.st_mtime_ns and host.stat().st_ino == made.st_ino
    own.write_text(own.read_text() + "// and more\n")
    (tmp_path / "stamp.txt").write_text(build._stamp() + "\n")
    build.build()
    assert host.stat().st_ino != made.st_ino or host.stat().st_mtime_ns != made.st_mtime_ns
    own.write_text(own.read_text() + "// and more\n")
    (tmp_path / "stamp.txt").write_text(build._stamp() + "\n")
    monkeypatch.setattr(build, "_no_extension", lambda: "no g++")
    build.build()
    assert host.is_file() and build.HostLibrary(ctypes.CDLL(None), (), (), {}) is not None and not build._host_is_current(tmp_path)
