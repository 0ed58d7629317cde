"""The build: what an installed package brings along, and what happens without the optional parts."""
import ctypes
import fnmatch
import re
import sysconfig
import tomllib
from pathlib import Path

import pytest

from ultraattn_b200 import _lib, build
from ultraattn_b200.ops import attention as A

ROOT = Path(build.__file__).resolve().parents[1]


def test_an_installed_package_brings_every_source():
    globs = tomllib.loads((ROOT / "pyproject.toml").read_text())["tool"]["setuptools"]["package-data"]["ultraattn_b200"]
    files = [f"csrc/{f.name}" for f in build.CSRC.iterdir() if f.is_file()]
    assert len(files) > 10
    assert [f for f in files if not any(fnmatch.fnmatch(f, g) for g in globs)] == []


@pytest.fixture
def host_dir(monkeypatch, tmp_path):
    _lib.load()
    monkeypatch.setattr(build, "HOST_PATH", tmp_path / "ua_host.so")
    monkeypatch.setattr(_lib, "_host", [])
    return tmp_path


def test_without_a_compiler_the_library_is_enough(host_dir, monkeypatch):
    """The host extension is left out with a warning, once, and calls go through Python."""
    monkeypatch.setenv("CXX", "no-such-compiler")
    lib = _lib.load()
    assert build._host_needs_build()
    with pytest.warns(UserWarning, match="through Python"):
        assert build.build_all() == build.LIB_PATH
    assert not build._host_needs_build() and build.host_path() is None
    assert _lib.host() is None and _lib.load() is lib
    monkeypatch.setattr(build, "_host_tools", lambda: "a compiler has been installed")
    assert build._host_needs_build()


def test_an_extension_that_does_not_load_is_left_out(host_dir):
    build.HOST_PATH.write_bytes(b"not a shared object")
    build._host_stamp().write_text(build.host_digest())
    with pytest.warns(UserWarning, match="through Python"):
        assert _lib.host() is None


def test_an_explicit_library_is_used_alone(host_dir, monkeypatch):
    monkeypatch.setattr(build, "host_path", lambda: pytest.fail("looked for the extension of another library"))
    monkeypatch.setenv("UA_LIB_PATH", str(build.LIB_PATH))
    assert _lib.host() is None


def test_an_extension_belongs_to_its_interpreter_flags_and_sources(host_dir, monkeypatch):
    build.HOST_PATH.write_bytes(b"")
    build._host_stamp().write_text(build.host_digest())
    assert build.host_path() == build.HOST_PATH
    get = sysconfig.get_config_var
    for change in (lambda m: m.setattr(sysconfig, "get_config_var", lambda n: "cpython-399" if n == "SOABI" else get(n)),
                   lambda m: m.setattr(build, "HOST_FLAGS", [*build.HOST_FLAGS, "-g"]), lambda m: m.setenv("CXX", "clang++"),
                   lambda m: m.setattr(build, "_torch_dir", lambda: host_dir)):
        (host_dir / "version.py").write_text("another PyTorch")
        with monkeypatch.context() as m:
            change(m)
            assert build.host_path() is None
    assert build.host_path() == build.HOST_PATH
    assert build.source_digest() == build.STAMP_PATH.read_text().strip()          # (the kernel library depends on none of it)


def test_argument_blocks_of_python_are_those_of_the_header():
    text = re.sub(r"//.*", "", (build.CSRC / "arg_blocks.h").read_text())
    fields = {}
    for name, body in re.findall(r"struct (\w+) \{(.*?)\n\};", text, re.S):
        fields[name] = []
        for kind, names in re.findall(r"([\w ]+\**)[ ]((?:\*?\w+(?:, )?)+);", body):
            for n in names.split(", "):
                inner = fields.get(kind.strip(), [""])
                fields[name] += [f"{n.lstrip('*')}.{i}".rstrip(".") for i in inner]
    for mirror in (_lib.UaTensorSrc, _lib.UaOutDst):
        assert [n for n, _ in mirror._fields_] == fields[mirror.__name__] and all(ctypes.sizeof(t) == 8 for _, t in mirror._fields_)
    assert A._DENSE_FWD.size == 8 * len(fields["UaDenseFwd"]) and A._LOCAL_BWD.size == 8 * len(fields["UaLocalBwd"])
    assert fields["UaLocalBwd"][28:] == ("o o_row_stride o_batch_stride lse dvec dq32 dq dk dv dkv_row_stride dkv_batch_stride cols segs "
                                         "tiles n_tiles dense skewed").split()          # (attn_bwd_local packs them in this order)
