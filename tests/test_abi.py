"""The C-ABI shared library loads on a GPU-less box and exports every symbol that
include/evo_b200.h declares (no compute calls here)."""
import ctypes
import os
import re

import pytest

from evo_b200 import _lib

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def header_functions():
    src = open(os.path.join(ROOT, "include", "evo_b200.h")).read()
    src = re.sub(r"/\*.*?\*/", "", src, flags=re.S)
    names = re.findall(r"\b(evo_[a-z0-9_]+)\s*\(", src)
    return sorted(set(names))


def test_library_is_built_in_tree():
    assert os.path.exists(_lib.LIB_PATH), "run `python -m evo_b200.build` (or __graft_entry__.build())"
    assert os.path.dirname(_lib.LIB_PATH) == os.path.join(ROOT, "evo_b200")


def test_every_declared_symbol_is_exported():
    names = header_functions()
    assert len(names) >= 18
    handle = ctypes.CDLL(_lib.LIB_PATH)
    missing = [n for n in names if not hasattr(handle, n)]
    assert not missing, f"declared in include/evo_b200.h but not exported: {missing}"


def test_binding_table_covers_the_header():
    assert sorted(_lib.SIGNATURES) == header_functions()


def test_loader_binds_and_reports_version():
    lib = _lib.lib()
    assert lib.evo_abi_version() == 1
    assert lib.evo_last_error() is not None
    lib.evo_reset_launch_count()
    assert lib.evo_launch_count() == 0


def test_missing_library_fails_loudly(monkeypatch, tmp_path):
    monkeypatch.setattr(_lib, "_lib", None)
    monkeypatch.setattr(_lib, "LIB_PATH", str(tmp_path / "nope.so"))
    with pytest.raises(_lib.EvoError, match="no CPU"):
        _lib.lib()


def test_header_is_plain_c_and_a_c_host_binds_every_entry_point(tmp_path):
    """include/evo_b200.h is the boundary for ANY host: it must compile as C99 and as C++ on its own, and a C program that
    #includes it and dlopen()s the library must resolve every declared entry point and get answers from the two that need no
    GPU (no torch, no Python anywhere near this binding)."""
    import shutil
    import subprocess
    gcc, gxx = shutil.which("gcc"), shutil.which("g++")
    if not gcc or not gxx:
        pytest.skip("gcc / g++ not available")
    hdr = os.path.join(ROOT, "include", "evo_b200.h")
    for cmd in ([gcc, "-std=c99", "-Wall", "-Wextra", "-pedantic", "-Werror", "-fsyntax-only", "-x", "c", hdr],
                [gxx, "-std=c++11", "-Wall", "-Wextra", "-Werror", "-fsyntax-only", "-x", "c++", hdr]):
        r = subprocess.run(cmd, capture_output=True, text=True)
        assert r.returncode == 0, r.stderr
    names = header_functions()
    src = tmp_path / "host.c"
    src.write_text(
        '#include <dlfcn.h>\n#include <stdio.h>\n#include "evo_b200.h"\n'
        "int main(int argc, char** argv) {\n"
        "  void* h = dlopen(argv[1], RTLD_NOW | RTLD_LOCAL);\n"
        '  if (!h) { fprintf(stderr, "dlopen: %s\\n", dlerror()); return 2; }\n'
        "  const char* names[] = {" + ", ".join(f'"{n}"' for n in names) + "};\n"
        "  int missing = 0;\n"
        "  for (unsigned i = 0; i < sizeof(names) / sizeof(names[0]); ++i) if (!dlsym(h, names[i])) { fprintf(stderr, \"missing %s\\n\", names[i]); ++missing; }\n"
        "  int (*version)(void) = (int (*)(void))dlsym(h, \"evo_abi_version\");\n"
        "  const char* (*last_error)(void) = (const char* (*)(void))dlsym(h, \"evo_last_error\");\n"
        '  printf("%d %d %s\\n", missing, version(), last_error() ? "str" : "null");\n'
        "  (void)argc; return missing != 0;\n}\n")
    exe = tmp_path / "host"
    r = subprocess.run([gcc, "-std=gnu99", "-I", os.path.join(ROOT, "include"), str(src), "-o", str(exe), "-ldl"], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([str(exe), _lib.LIB_PATH], capture_output=True, text=True)
    assert r.returncode == 0 and r.stdout.split() == ["0", "1", "str"], (r.stdout, r.stderr)


def test_error_convention_without_a_gpu():
    """No exception crosses the ABI: a rejected argument returns a negative code and leaves the reason in evo_last_error() before
    anything is launched (so this runs on a GPU-less box); and a well-formed call on a box without a GPU FAILS, loudly, with the
    CUDA runtime's reason -- there is no CPU path to fall back to."""
    import torch
    if torch.cuda.is_available():
        pytest.skip("this is the GPU-less half of the error convention")
    lib = _lib.lib()
    p = _lib.GemmParams(A=0x1000, lda=100, W=0x2000, C=0x3000, ldc=64, bias=None, residual=None, ldr=64, M=4, N=64, K=100, epilogue=0, variant=0)
    assert lib.evo_gemm(ctypes.byref(p), None) < 0 and b"K (100) must be a multiple of 64" in lib.evo_last_error()
    assert lib.evo_sample(None, None, 2, 2000, 1, 0.0, 1.0, 0, 0, None) < 0 and b"vocabulary 2000 unsupported" in lib.evo_last_error()
    assert lib.evo_kv_append(None, None, 1, 10, 2, 128, 10, 16, None) < 0 and b"exceeds the KV cache (16)" in lib.evo_last_error()   # mha.py:367
    with pytest.raises(_lib.EvoError, match="exceeds the KV cache"):
        _lib.check(lib.evo_kv_append(None, None, 1, 10, 2, 128, 10, 16, None), "evo_kv_append")
    rc = lib.evo_rmsnorm(ctypes.c_void_p(0x1000), ctypes.c_void_p(0x2000), ctypes.c_void_p(0x3000), 4, 4096, 1e-6, None)
    assert rc < 0 and b"failed" in lib.evo_last_error()


def _workspace_in_a_process(code):
    """Workspace queries are host arithmetic; one that divides by zero would take this process along."""
    import subprocess
    import sys
    r = subprocess.run([sys.executable, "-c", "import ctypes as C\nfrom evo_b200 import _lib\nfrom evo_b200._lib import *\nlib = _lib.lib()\n" + code],
                       cwd=ROOT, capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, f"ended with {r.returncode}: {r.stderr[-500:]}"
    return [int(x) for x in r.stdout.split()]


def test_gated_delta_workspace_of_an_empty_call_is_empty():
    got = _workspace_in_a_process(
        "for B, H, L in ((0, 4, 64), (0, 4, 16), (0, 4, 5000), (1, 0, 64), (-1, 4, 64), (2, 4, 64)):\n"
        "    print(lib.evo_gated_delta_workspace(C.byref(GatedDeltaParams(B=B, L=L, H=H, G=1, dk=128, dv=128, ld=384, dtype=0))))\n")
    assert got[:5] == [0] * 5 and got[5] > 0


def test_hyena_workspace_of_an_empty_call_is_empty():
    got = _workspace_in_a_process(
        "for B, L in ((0, 64), (0, 500), (0, 2000), (-1, 500), (1, 0), (1, 500)):\n"
        "    print(lib.evo_hyena_fwd_workspace(C.byref(HyenaParams(B=B, L=L, D=512, S=8, nheads=4))))\n")
    assert got[:5] == [0] * 5 and got[5] > 0


def test_lost_waits_are_none_and_their_limit_belongs_to_the_thread():
    import threading
    lib = _lib.lib()
    assert lib.evo_lost_waits(1) == 0
    _lib.check_lost_waits()
    default = lib.evo_set_wait_polls(5)
    seen = []
    t = threading.Thread(target=lambda: seen.append(lib.evo_set_wait_polls(7)))
    t.start()
    t.join()
    assert seen == [default] and default > 1 << 16
    assert lib.evo_set_wait_polls(-1) == 5 and lib.evo_set_wait_polls(default) == default


def test_short_gated_delta_calls_go_token_by_token_where_that_is_faster():
    """The line between the token-by-token kernel (no workspace, or fp32 read-outs) and the 64-token blocks (their matrices, 32 KB each, as well)."""
    lib = _lib.lib()

    def blocks(pairs, dk, dv, L):
        p = _lib.GatedDeltaParams(B=pairs // 8, L=L, H=8, G=8, dk=dk, dv=dv, ld=8 * (2 * dk + dv), dtype=0)
        return lib.evo_gated_delta_workspace(ctypes.byref(p)) > 4 * pairs * L * dv + 32768 * pairs
    for pairs, dk, dv, first in ((8, 64, 64, 48), (32, 128, 128, 48), (128, 64, 128, 48), (256, 128, 64, 48), (512, 64, 64, 32), (2048, 128, 128, 32), (8, 128, 16, 32), (128, 64, 32, 32),
                                 (512, 128, 16, 48), (1024, 128, 16, 128), (1024, 64, 32, 48)):
        assert not blocks(pairs, dk, dv, first - 1) and blocks(pairs, dk, dv, first), (pairs, dk, dv, first)
