"""The build: what an installed package brings along, and what happens without the optional parts."""
import fnmatch
import tomllib
from pathlib import Path

from ultraattn_b200 import build

ROOT = Path(build.__file__).resolve().parents[1]


def test_an_installed_package_brings_every_source():
    globs = tomllib.loads((ROOT / "pyproject.toml").read_text())["tool"]["setuptools"]["package-data"]["ultraattn_b200"]
    files = [f"csrc/{f.name}" for f in build.CSRC.iterdir() if f.is_file()]
    assert len(files) > 10
    assert [f for f in files if not any(fnmatch.fnmatch(f, g) for g in globs)] == []
