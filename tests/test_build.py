"""The build's record of what made an object: another command line makes it stale, as a newer source does, so that
no library mixes objects of different flags; and the flags keep each unit in one piece."""

from __future__ import annotations

import importlib.util
import os
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]


@pytest.fixture()
def build():
    spec = importlib.util.spec_from_file_location("qoraholo_b200_build", ROOT / "qoraholo_b200" / "_build.py")
    mod = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(mod)
    return mod


def test_other_flags_make_an_object_stale(build, tmp_path):
    src, obj = tmp_path / "a.cpp", tmp_path / "a.o"
    src.write_text("int a() { return 1; }\n")

    def command(*flags):
        return ["g++", *flags, "-MD", "-MF", str(obj.with_suffix(".d")), "-c", str(src), "-o", str(obj)]

    assert build._stale(obj, src, command("-O1"))
    build._compile(command("-O1"))
    assert not build._stale(obj, src, command("-O1"))
    assert build._stale(obj, src, command("-O2"))
    assert build._stale(obj, src, command("-O1", "-DX"))
    src.write_text("int a( {\n")  # a compile that fails leaves nothing that passes for up to date
    with pytest.raises(RuntimeError):
        build._compile(command("-O1"))
    old = obj.stat().st_mtime - 10
    os.utime(src, (old, old))
    assert build._stale(obj, src, command("-O1"))


def test_units_are_optimised_whole(build):
    assert not any("split-compile" in flag for flag in build.NVCC_FLAGS)
