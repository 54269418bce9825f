"""The C-ABI library loads without a GPU and exports every symbol that
include/evoattn.h declares; argument validation returns codes."""
import ctypes as C
import os
import re

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _declared_symbols():
    src = open(os.path.join(ROOT, "include", "evoattn.h")).read()
    src = re.sub(r"/\*.*?\*/", "", src, flags=re.S)
    return sorted(set(re.findall(r"\b(evo_[a-z0-9_]+)\s*\(", src)))


def test_header_symbols_exported():
    import _evoattn
    names = _declared_symbols()
    assert "evo_fwd" in names and "evo_bwd" in names and len(names) >= 8
    h = C.CDLL(_evoattn.LIB_PATH)
    for n in names:
        assert hasattr(h, n), f"{n} declared in include/evoattn.h but not exported"
    # and the binding covers them all
    assert sorted(_evoattn.SYMBOLS) == names


def test_version_is_the_header_s():
    import _evoattn
    src = open(os.path.join(ROOT, "include", "evoattn.h")).read()
    declared = int(re.search(r"#define EVO_ABI_VERSION (\d+)", src).group(1))
    assert _evoattn.lib().evo_version() == declared == _evoattn.ABI_VERSION
    # what each minor version added since 103
    assert declared >= 104 and "evo_bwd_ex" in _declared_symbols()


def test_version_and_strerror():
    import _evoattn
    lib = _evoattn.lib()
    assert lib.evo_version() // 100 == 1
    assert _evoattn.strerror(0) == "ok"
    assert "dimensions" in _evoattn.strerror(-1)
    assert _evoattn.strerror(-12345) == "unknown error"


def test_argument_validation_without_gpu():
    import _evoattn
    lib = _evoattn.lib()
    good = _evoattn.EvoDims(1, 4, 128, 2, 32)
    assert lib.evo_bwd_workspace_bytes(C.byref(good)) > 4 * 4 * 128 * 2 * 32
    for bad in (_evoattn.EvoDims(1, 4, 128, 2, 256), _evoattn.EvoDims(1, 4, 100, 2, 32),
                _evoattn.EvoDims(0, 4, 128, 2, 32), _evoattn.EvoDims(1, 4, 128, 2, 48), _evoattn.EvoDims(1, 4, 128, 2, 8)):
        assert lib.evo_bwd_workspace_bytes(C.byref(bad)) == 0
        rc = lib.evo_fwd(C.byref(bad), 16, 16, 16, 16, 16, 16, None, 16, 0.0, None)
        assert rc == -1
    assert lib.evo_fwd(C.byref(good), None, 16, 16, 16, 16, 16, None, 16, 0.0, None) == -2
    assert lib.evo_fwd(C.byref(good), 8, 16, 16, 16, 16, 16, None, 16, 0.0, None) == -3
    assert lib.evo_fwd(C.byref(good), 16, 16, 16, 16, 16, 16, 8, 16, 0.0, None) == -3    # o_resid misaligned
    assert lib.evo_fwd(None, 16, 16, 16, 16, 16, 16, None, 16, 0.0, None) == -2
    args = [16] * 13
    assert lib.evo_bwd(C.byref(good), *args, 256, 0, 0.0, None) == -4    # workspace too small
    assert lib.evo_selftest_mma(48, 16, 16, 16, 16, 16, 16, 16, None) == -1


def test_missing_library_fails_loudly(monkeypatch):
    import _evoattn
    monkeypatch.setattr(_evoattn, "_lib", None)
    monkeypatch.setattr(_evoattn, "LIB_PATH", "/nonexistent/libevoattn.so")
    with pytest.raises(ImportError):
        _evoattn.lib()


def _bytes_of_n_rows(d):
    """Workspace whose fp32 dQ area holds N rows per (row of S, head), without rounding N up."""
    up = lambda x: -(-x // 256) * 256
    bs, ntp, dh = d.B * d.S, -(-d.N // 128) * 128, 32 if d.D <= 32 else 64 if d.D <= 64 else 128
    return up(up(up(bs * d.H * ntp * 16) + bs * ntp * 16) + bs * d.N * d.H * dh * 4)


def test_static_scratch_takes_what_fits_without_rounding():
    """The rounding of N in evo_bwd_workspace_bytes does not shrink what the fixed scratch array takes."""
    import _evoattn
    lib = _evoattn.lib()
    cap = lib.evo_bwd_static_scratch_capacity()
    for n, d in ((40, 32), (136, 64), (264, 128)):
        h = 4
        s = max(s for s in range(1, 4096) if _bytes_of_n_rows(_evoattn.EvoDims(1, s, n, h, d)) <= cap)
        dims = _evoattn.EvoDims(1, s, n, h, d)
        assert lib.evo_bwd_workspace_bytes(C.byref(dims)) > cap
        nulls = [None] * 13
        assert lib.evo_bwd_static_scratch(C.byref(dims), *nulls, 0.0, None) != -9      # (a null pointer, or no device)
        dims = _evoattn.EvoDims(1, s + 1, n, h, d)
        assert lib.evo_bwd_static_scratch(C.byref(dims), *nulls, 0.0, None) == -9
