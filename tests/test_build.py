"""The two build products: the C library, which needs nvcc alone, and the Python extension of eager calls, which is optional."""
import subprocess

import pytest

from nanoserve_b200 import build, ops


def compilers(monkeypatch, tmp_path, gxx):
    """Builds go to tmp_path; the compilers are replaced: nvcc succeeds, g++ does what `gxx` does.  Returns their command lines."""
    monkeypatch.setattr(build, "LIB_DIR", str(tmp_path))
    monkeypatch.setattr(build, "LIB_PATH", str(tmp_path / "libnanoserve.so"))
    monkeypatch.setattr(build, "CALL_PATH", str(tmp_path / "nanoserve_call.so"))
    ran = []

    def run(cmd, **kw):
        ran.append(cmd)
        return gxx(cmd) if cmd[0] == "g++" else subprocess.CompletedProcess(cmd, 0, "", "")

    monkeypatch.setattr(build.subprocess, "run", run)
    return ran


def no_compiler(cmd):
    raise FileNotFoundError(2, "No such file or directory", cmd[0])


def no_header(cmd):
    return subprocess.CompletedProcess(cmd, 1, "", "fatal error: Python.h: No such file or directory")


@pytest.mark.parametrize("gxx", [no_compiler, no_header])
def test_the_library_is_built_without_the_extension(monkeypatch, tmp_path, capsys, gxx):
    ran = compilers(monkeypatch, tmp_path, gxx)
    assert build.build() == build.LIB_PATH
    assert [c[0] for c in ran] == [build.os.environ.get("NVCC", "nvcc"), "g++"]
    assert "nanoserve_call.so was not built" in capsys.readouterr().err


def test_an_extension_that_does_not_load_is_left_out(monkeypatch, tmp_path):
    monkeypatch.setattr(ops, "_LIB_DEFAULT", str(tmp_path / "libnanoserve.so"))
    assert ops._load_call() == (None, None)  # not built
    (tmp_path / "nanoserve_call.so").write_bytes(b"\x7fELF, cut off")
    (tmp_path / "nanoserve_call.so.built_for").write_text(build.built_for())
    with pytest.warns(RuntimeWarning, match="does not load"):
        assert ops._load_call() == (None, None)


def test_the_extension_follows_torch_and_python(monkeypatch, tmp_path):
    """Built again where its note names another torch or Python, never loaded there, and never there in part."""
    written = []

    def gxx(cmd):
        out = cmd[cmd.index("-o") + 1]
        written.append(out)
        open(out, "wb").close()
        return subprocess.CompletedProcess(cmd, 0, "", "")

    ran = compilers(monkeypatch, tmp_path, gxx)
    build.build_call()
    build.build_call()
    assert len(ran) == 1 and build.call_matches(build.CALL_PATH)
    monkeypatch.setattr(build, "built_for", lambda: "torch 0.0 cpython-00")
    monkeypatch.setattr(ops, "_LIB_DEFAULT", build.LIB_PATH)
    with pytest.warns(RuntimeWarning, match="another torch or Python"):
        assert ops._load_call() == (None, None)
    build.build_call()
    assert len(ran) == 2 and build.call_matches(build.CALL_PATH)
    assert build.CALL_PATH not in written
    assert sorted(p.name for p in tmp_path.iterdir()) == ["nanoserve_call.so", "nanoserve_call.so.built_for"]


def test_an_extension_built_after_the_import_is_used(monkeypatch, lib_path):
    """A clean checkout: the tests' modules import ops before the fixture builds anything."""
    if not build.os.path.exists(build.CALL_PATH):
        pytest.skip("the extension cannot be built here")
    monkeypatch.setattr(ops, "_call_linear", None)
    monkeypatch.setattr(ops, "_call_quantize", None)
    k = ops.Kernels(lib_path)
    assert k._linear is not None and k._quantize is not None
    assert ops._call_linear is not None and ops._call_quantize is not None
