"""What the build and the front end do where torch, a compiler or the native front end is missing."""
import builtins
import sys
import types

import pytest

from antares_b200 import _lib, build


def test_the_library_does_not_need_torch(monkeypatch):
    real = builtins.__import__

    def no_torch(name, *args, **kw):
        if name == "torch" or name.startswith("torch."):
            raise ImportError("no torch here")
        return real(name, *args, **kw)
    monkeypatch.setattr(builtins, "__import__", no_torch)
    monkeypatch.setattr(build, "up_to_date", lambda: True)
    assert build.build() == build.LIB and build.build_fastcall() is None


def test_the_library_does_not_need_a_host_compiler(monkeypatch, tmp_path):
    monkeypatch.setenv("CXX", str(tmp_path / "no-such-compiler"))
    monkeypatch.setattr(build, "FAST", str(tmp_path / "_fastcall.so"))
    monkeypatch.setattr(build, "up_to_date", lambda: True)
    assert build.build() == build.LIB


def test_another_torch_means_another_build(monkeypatch, tmp_path):
    """A front end newer than its source is still rebuilt when it was built for another torch."""
    made = []
    fast = tmp_path / "_fastcall.so"
    fast.write_bytes(b"")

    def compiler(cmd):
        made.append(cmd)
        open(cmd[cmd.index("-o") + 1], "w").close()
    monkeypatch.setattr(build, "FAST", str(fast))
    monkeypatch.setattr(build.subprocess, "check_call", compiler)
    (tmp_path / "_fastcall.so.built_for").write_text("torch 0.1, python 3")
    build.build_fastcall()
    build.build_fastcall()
    assert len(made) == 1


@pytest.mark.parametrize("module", [None, types.SimpleNamespace(built_for=lambda: "torch 0.1, python 3", bind=lambda d: pytest.fail("bound"))])
def test_operators_run_without_the_native_front_end(monkeypatch, module):
    import antares_b200
    monkeypatch.setattr(_lib, "_fast", None)
    monkeypatch.setitem(sys.modules, "antares_b200._fastcall", module)  # None: cannot be imported
    if module is None:
        monkeypatch.delattr(antares_b200, "_fastcall", raising=False)
    else:
        monkeypatch.setattr(antares_b200, "_fastcall", module, raising=False)
    with pytest.warns(UserWarning, match="_fastcall.so is not used"):
        front = _lib.fast()
    assert front.w4a16(0, 1, 2, 3) is None and front.run(front.program(), 1) is None
    assert _lib.fast() is front
