"""The build of the native libraries (CPU): what is optional stops nothing."""
import shutil
import subprocess
import sys
from pathlib import Path

import pytest

from allie_b200 import PY_LIBRARY, build

ROOT = Path(__file__).resolve().parent.parent


def test_an_installed_copy_has_every_source(tmp_path):
    tree = tmp_path / "tree"
    tree.mkdir()
    for name in ("allie_b200", "src"):
        shutil.copytree(ROOT / name, tree / name, ignore=shutil.ignore_patterns("lib", "__pycache__"))
    for name in ("setup.py", "pyproject.toml"):
        shutil.copy(ROOT / name, tree / name)
    subprocess.run([sys.executable, "setup.py", "-q", "build_py", "--build-lib", str(tmp_path / "out")], cwd=tree, check=True,
                   capture_output=True)
    sources = [p.relative_to(ROOT) for p in build.CSRC.rglob("*") if p.is_file()]
    assert sources and all((tmp_path / "out" / p).is_file() for p in sources)


@pytest.mark.parametrize("trouble", ["no source", "no source, built before", "does not compile", "no compiler"])
def test_the_optional_library_does_not_stop_the_build(trouble, tmp_path, monkeypatch):
    csrc, lib = tmp_path / "csrc", tmp_path / "lib"
    (csrc / "py").mkdir(parents=True)
    lib.mkdir()
    if not trouble.startswith("no source"):
        (csrc / "py" / "tokens.cpp").write_text("not C++\n")
    for name, value in (("CSRC", csrc), ("LIB", lib), ("OBJ", lib / "obj")):
        monkeypatch.setattr(build, name, value)
    if trouble == "no source, built before":
        (lib / PY_LIBRARY).write_bytes(b"")
    if trouble == "no compiler":
        monkeypatch.setenv("CXX", str(tmp_path / "none"))
    built = []
    monkeypatch.setattr(build, "build_host", lambda *a: built.append("host"))
    monkeypatch.setattr(build, "build_cuda", lambda *a: built.append("cuda"))
    build.build_all()
    assert built == ["host", "cuda"]
    assert (build.build_py() is None) == (trouble != "no source, built before")


@pytest.mark.parametrize("suffix", [".cpython-311-x86_64-linux-gnu.so", ".cpython-313t-x86_64-linux-gnu.so"])
def test_a_library_of_another_interpreter_is_not_loaded(suffix, monkeypatch):
    """It reads object layouts that are compiled in; the Python statement of the rules serves until there is one."""
    from allie_b200 import data

    if build.build_py() is None:
        pytest.skip("no interpreter headers")
    data._native_tokens.cache_clear()
    try:
        assert data._native_tokens() is not None
        data._native_tokens.cache_clear()
        monkeypatch.setattr("allie_b200.PY_LIBRARY", "liballie_py" + suffix)
        assert data._native_tokens() is None
    finally:
        data._native_tokens.cache_clear()
