"""What the build does with what it finds: a reference folder without sources,
objects older than a header."""
import os

import pytest

import oracle
from dtcf_gb300 import build


def test_an_empty_reference_folder_builds_the_restatement_alone(tmp_path, monkeypatch):
    monkeypatch.setenv("DTCF_REFERENCE", str(tmp_path))
    oracle.build(ref=True)


@pytest.mark.parametrize("header", ["a.h", "a.cuh"])
def test_an_object_older_than_a_header_is_compiled_again(tmp_path, monkeypatch, header):
    (tmp_path / "nvcc").write_text('#!/bin/sh\nfor last; do :; done\necho made >> "$last"\n')
    (tmp_path / "nvcc").chmod(0o755)
    for name in ("a.cu", header):
        (tmp_path / name).write_text("")
    for name, value in (("CSRC", tmp_path), ("OBJ", tmp_path), ("NVCC", tmp_path / "nvcc")):
        monkeypatch.setattr(build, name, str(value))
    src = str(tmp_path / "a.cu")
    obj, _ = build._compile(src, False)
    build._compile(src, False)
    assert open(obj).read() == "made\n"
    later = os.path.getmtime(obj) + 10
    os.utime(tmp_path / header, (later, later))
    build._compile(src, False)
    assert open(obj).read() == "made\nmade\n"
