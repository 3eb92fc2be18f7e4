"""Server.submit's two ways to the library (the native module, ctypes where it
is not built) hand over the same arguments and raise on the same inputs. The
library's function is a recorder here, so no GPU is needed."""

from __future__ import annotations

import ctypes as C

import numpy as np
import pytest
import torch

from atkdsp_b200 import serve

ARGS = [C.c_void_p, C.c_int, C.c_void_p, C.c_size_t, C.c_void_p, C.c_size_t, C.c_uint64, C.c_double]


@pytest.fixture
def server():
    """A Server over a recording function: (server, calls)."""
    calls = []

    def record(*a):
        calls.append(a)
        return -3 if a[1] == 7 else 0

    fn = C.CFUNCTYPE(C.c_int, *ARGS)(record)
    srv = serve.Server.__new__(serve.Server)
    srv._lib = type("L", (), {"atkdsp_server_submit": staticmethod(fn),
                              "atkdsp_server_destroy": staticmethod(lambda s: None)})
    srv._s, srv._submit = 4096, C.cast(fn, C.c_void_p).value
    return srv, calls


def _both(srv, calls, monkeypatch, *a, **k):
    got = []
    for native in (serve._native, None):
        monkeypatch.setattr(serve, "_native", native)
        calls.clear()
        try:
            got.append((srv.submit(*a, **k), list(calls)))
        except Exception as e:  # noqa: BLE001
            got.append((type(e), list(calls)))
    assert got[0] == got[1]
    return got[0]


@pytest.mark.parametrize("sid,tag,t", [(0, 0, 0.0), (7, 2**64 - 1, 1e9), (-1, -1, 3), (np.int64(5), np.uint32(9), np.float32(2)),
                                       (2**31 + 3, 2**70 + 5, -0.0), (True, 1.9, "4.5")])
@pytest.mark.parametrize("dtype,n", [(torch.complex64, 12), (torch.int16, 12), (torch.int16, 13), (torch.complex64, 0)])
def test_same_arguments(server, monkeypatch, sid, tag, t, dtype, n):
    if serve._native is None:
        pytest.skip("the module was not built for this Python")
    srv, calls = server
    x, y = torch.zeros(n + 4, dtype=dtype)[4:], torch.zeros(3, 5, dtype=torch.complex64)
    rc, seen = _both(srv, calls, monkeypatch, sid, x, y, tag, t_arrival=t)
    assert len(seen) == 1 and rc == (-3 if int(sid) == 7 else 0)
    assert seen[0][3] == (n if dtype == torch.complex64 else n // 2) and seen[0][5] == 15


@pytest.mark.parametrize("bad", [dict(sid=None), dict(sid="x"), dict(block=3), dict(out=None), dict(tag=None),
                                 dict(t_arrival="soon"), dict(t_arrival=None)])
def test_same_refusals(server, monkeypatch, bad):
    if serve._native is None:
        pytest.skip("the module was not built for this Python")
    srv, calls = server
    a = dict(sid=0, block=torch.zeros(4, dtype=torch.int16), out=torch.zeros(4, dtype=torch.complex64), tag=0,
             t_arrival=0.0)
    a.update(bad)
    rc, seen = _both(srv, calls, monkeypatch, **a)
    assert isinstance(rc, type) and issubclass(rc, Exception) and not seen


@pytest.mark.parametrize("version", ["0x030B00F0", "0x030900F0", None])
def test_module_is_left_out_where_it_does_not_build(tmp_path, version):
    """Headers of a Python before 3.12 (declaring all the module uses), or a
    compiler that fails: make goes on, an older module is taken away, and the
    package's loader falls back to ctypes."""
    import shutil
    import subprocess
    from pathlib import Path
    src = Path(serve.__file__).resolve().parent
    (tmp_path / "csrc" / "py").mkdir(parents=True)
    (tmp_path / "lib").mkdir()
    shutil.copy(src / "Makefile", tmp_path / "Makefile")
    shutil.copy(src / "csrc" / "py" / "submit.c", tmp_path / "csrc" / "py" / "submit.c")
    so = tmp_path / "lib" / "_atkdsp_submit.so"
    so.write_bytes(b"stale")
    import os
    os.utime(so, (1, 1))
    args = ["make", "-C", str(tmp_path), str(so)]
    if version is None:
        args.append("HCC=false")
    else:
        import sysconfig
        (tmp_path / "inc").mkdir()
        (tmp_path / "inc" / "Python.h").write_text(
            f'#include "{sysconfig.get_paths()["include"]}/Python.h"\n#undef PY_VERSION_HEX\n#define PY_VERSION_HEX {version}\n')
        args.append(f"PY_INC={tmp_path / 'inc'} -I{sysconfig.get_paths()['include']}")
    r = subprocess.run(args, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    assert not so.exists()
