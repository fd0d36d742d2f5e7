"""The C ABI library loads without a GPU and exports every function that
include/adz_b200.h declares; calls that need a device fail with a status, not
a crash."""
import ctypes as C
import os
import re

import numpy as np
import pytest
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
HEADER = os.path.join(ROOT, "include", "adz_b200.h")


def declared_functions():
    src = open(HEADER).read()
    src = re.sub(r"/\*.*?\*/", "", src, flags=re.S)
    names = re.findall(r"^\s*(?:const\s+)?[A-Za-z_][\w\s\*]*?\b([A-Za-z_]\w*)\s*\(", src, flags=re.M)
    return sorted(set(n for n in names if n not in ("if", "while", "return", "sizeof")))


@pytest.fixture(scope="module")
def L():
    from gem_b200 import build
    build.build()
    from gem_b200 import adz
    return adz.lib()


def test_header_symbols_exported(L):
    names = declared_functions()
    assert len(names) >= 20
    for n in names:
        assert hasattr(L, n), n


def test_reference_symbol_set_present(L):
    for n in ("Vsearch_setup", "Vsearch_setup_plus", "Tricublin_zyx1_n", "Tricublin_zyx1_n_m", "Tricublin_zyx1_m_n",
              "Tricublin_zyx1_p", "Tricublin_mono_zyx_n", "Tricublin_mono_zyx_n_m", "Tricublin_mono_zyx_m_n",
              "Tricublin_zyx3_n"):
        assert hasattr(L, n)


def test_errors_without_device(L):
    from gem_b200 import adz, synth
    if torch.cuda.is_available():
        pytest.skip("device present")
    with pytest.raises(adz.AdzError) as e:
        adz.Adz.from_config(synth.config_small(32, 32, 10))
    assert e.value.status in (8, 2)
    assert L.adzc_error_string(8) == b"no CUDA device"
    # argument checks come before any device work
    assert L.adzc_setup(None, None) == 1
    assert L.adzc_traject(None, 0, C.c_double(1.0), 1, *([None] * 9)) == 1
    assert L.adzc_tricub(None, 0, 0, 0, None, None, None, None, None, None, None) == 1
    # a tile whose extended volume needs offsets beyond 32 bits is refused
    g = adz.AdzcGrid()
    big = np.zeros(64)
    g.ni, g.nj, g.nk, g.maxcfl = 60000, 60000, 4, 3
    g.zm = g.zt = g.zx = g.cy = big.ctypes.data_as(C.POINTER(C.c_double))
    h = C.c_void_p()
    assert L.adzc_setup(C.byref(g), C.byref(h)) == 9
    lev = np.linspace(3000.0, 100.0, 3)
    out = C.c_void_p()
    assert L.adzc_ztab_create(lev.ctypes.data, 3, 10, 10, 0, 0, C.byref(out)) == 3  # nk < 4


def test_boundary_flux_copies(L):
    """Which tracers of a boundary-flux call are read from copies, and how many
    copies exist at a time (groups of 8 tracers)."""
    ext = 4096

    def plan(srcs, fo, fi):
        n = len(srcs)
        arr = lambda v: (C.c_void_p * n)(*v)  # noqa: E731
        when = (C.c_ubyte * n)()
        f = L.adz_internal_flux_copies
        f.argtypes = [C.c_int] + [C.c_void_p] * 3 + [C.c_size_t, C.c_void_p]
        return f(n, arr(srcs), arr(fo), arr(fi), ext, when), list(when)

    at = lambda q: 0x10000 + q * ext  # noqa: E731
    n = 19
    src, fo, fi = ([at(100 * b + q) for q in range(n)] for b in range(3))
    assert plan(src, fo, fi) == (0, [0] * n)
    # a tracer in its own flux array, one that overlaps it by a byte, one that only touches it
    s = list(src)
    s[1], s[2], s[3] = fo[1], fi[2] + ext - 1, fo[n - 1] + ext
    assert plan(s, fo, fi) == (2, [0, 1, 1] + [0] * 16)
    # the largest group decides: one copy in the first, three in the second
    s = list(src)
    s[0], s[8], s[9], s[15] = fo[0], fo[9], fi[8], fo[15]
    assert plan(s, fo, fi) == (3, [1] + [0] * 7 + [1, 1] + [0] * 5 + [1] + [0] * 3)
    # an array of an earlier group; an array of a later group is written after the tracer was read
    s = list(src)
    s[17], s[18], s[3], s[4] = fi[0], fo[16], fo[18], None
    got = plan(s, fo, fi)
    assert got[0] == 2 and [got[1][q] for q in (3, 4, 17, 18)] == [0, 0, 2, 1]


def test_no_library_no_fallback(monkeypatch, tmp_path):
    """Without the built library every entry point raises: there is no CPU
    fallback behind the binding."""
    from gem_b200 import adz, synth
    monkeypatch.setattr(adz, "LIB_PATH", str(tmp_path / "missing.so"))
    monkeypatch.setattr(adz, "_LIB", None)
    with pytest.raises(FileNotFoundError):
        adz.lib()
    with pytest.raises(FileNotFoundError):
        adz.Adz.from_config(synth.config_small(16, 16, 8))
