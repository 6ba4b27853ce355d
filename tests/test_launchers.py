"""Launchers called through csrc/fastcall.c: every kind of parameter arrives where ctypes would put it, and what it does not take goes to
ctypes as before."""

import ctypes
import os
import subprocess

import pytest

from tandemllm_b200.kernels import build

SOURCE = """
long long whole[32]; float real[8];
int mixed(void* a, long long b, float x, void* c, int d, unsigned e, float y, int f, void* g, long long h, int i, float z, int j) {
  whole[0] = (long long)a; whole[1] = b; whole[2] = (long long)c; whole[3] = d; whole[4] = e; whole[5] = f; whole[6] = (long long)g;
  whole[7] = h; whole[8] = i; whole[9] = j; real[0] = x; real[1] = y; real[2] = z;
  return d - j;
}
int none(void) { return 7; }
"""


@pytest.fixture(scope="module")
def library(tmp_path_factory):
    folder = tmp_path_factory.mktemp("fastcall")
    (folder / "l.c").write_text(SOURCE)
    subprocess.run(["cc", "-O1", "-shared", "-fPIC", str(folder / "l.c"), "-o", str(folder / "l.so")], check=True)
    lib = ctypes.CDLL(str(folder / "l.so"))
    P, L, I, U, F = ctypes.c_void_p, ctypes.c_longlong, ctypes.c_int, ctypes.c_uint, ctypes.c_float
    lib.mixed.argtypes, lib.mixed.restype = [P, L, F, P, I, U, F, I, P, L, I, F, I], I
    return lib


@pytest.mark.skipif(build.build_fastcall() is None, reason="no C compiler or another platform")
def test_arguments_of_every_kind_arrive_as_through_ctypes(library):
    fast = build.Launchers(library, ["mixed"])
    assert type(fast.mixed).__name__ == "Launcher" and fast.mixed.restype is ctypes.c_int and len(fast.mixed.argtypes) == 13
    cases = [(1 << 47, -5, 1.5, None, -7, 8, 2.5, 9, 123, 1 << 40, -11, 3, 13), (None, 2 ** 63 - 1, -0.0, 2 ** 64 - 1, 2 ** 31, 2 ** 32 + 3, 1e30, True, 0, -1, 0, False, -1)]
    for args in cases:
        seen = []
        for lib in (library, fast):
            code = lib.mixed(*args)
            seen.append((code, list((ctypes.c_longlong * 32).in_dll(library, "whole")), [f.hex() for f in (ctypes.c_float * 8).in_dll(library, "real")]))
        assert seen[0] == seen[1]
    assert fast.mixed(ctypes.c_void_p(5), 0, 0.0, None, 1, 0, 0.0, 0, None, 0, 0, 0.0, 0) == 1          # (ctypes takes the wrapped pointer)
    assert (ctypes.c_longlong * 32).in_dll(library, "whole")[0] == 5
    for bad in ((1, 2), cases[0][:2] + ("x",) + cases[0][3:], cases[0][:4] + ("x",) + cases[0][5:]):
        with pytest.raises((TypeError, ctypes.ArgumentError)):
            fast.mixed(*bad)
    assert fast.none() == 7                                                                              # (no declared parameters)


def launched_through(libraries):
    """(functions with declared parameters that return an int, those of them that go through the extension)"""
    fit, through = [], []
    for lib in libraries:
        for name, fn in vars(lib._library).items():
            if name.startswith("tl_") and fn.argtypes and fn.restype is ctypes.c_int:
                fit.append(name)
                if name in vars(lib):
                    assert type(vars(lib)[name]).__name__ == "Launcher"
                    through.append(name)
    return fit, through


def test_the_kernel_libraries_are_called_through_it_where_it_was_built():
    from tandemllm_b200.kernels import ops, tensorcore
    fit, through = launched_through([ops.core(), tensorcore.lib()])
    assert len(fit) > 60
    if build.build_fastcall() is None:
        assert not through
    else:
        assert sorted(set(fit) - set(through)) == []


@pytest.mark.parametrize("broken", ["compiler fails", "compiler cannot run", "file is no extension"])
def test_launches_go_through_ctypes_where_the_extension_cannot_be_had(broken, library, tmp_path, monkeypatch):
    cc = tmp_path / "cc"
    cc.write_text("#!/bin/sh\nexit 1\n" if broken == "compiler fails" else
                  "#!/no/such/shell\n" if broken == "compiler cannot run" else
                  '#!/bin/sh\nfor a in "$@"; do o=$a; done\necho no > "$o"\n')
    cc.chmod(0o755)
    monkeypatch.setenv("PATH", f"{tmp_path}:{os.environ['PATH']}")
    monkeypatch.setattr(build, "build_dir", lambda: str(tmp_path))            # (where no extension has been built)
    monkeypatch.setattr(build, "_launcher", None)
    plain = build.Launchers(library, ["mixed"])
    assert "mixed" not in vars(plain) and plain.mixed(None, 0, 0.0, None, 5, 0, 0.0, 0, None, 0, 0, 0.0, 3) == 2
    assert not [f for f in os.listdir(tmp_path) if f.endswith(".so")] or broken == "file is no extension"
