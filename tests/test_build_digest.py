"""The hash that names a compiled library: of its sources, its flags and every header, and headers that have not
changed are read once per process."""

import hashlib
import os
from pathlib import Path


def test_headers_are_read_once_until_one_changes(tmp_path, monkeypatch):
    from scratch_llm_b200.kernels import build
    (tmp_path / "a.cuh").write_text("one")
    (tmp_path / "b.h").write_text("two")
    (tmp_path / "k.cu").write_text("kernel")
    monkeypatch.setattr(build, "CSRC", tmp_path)
    monkeypatch.setattr(build, "_headers", None)
    read, read_bytes = [], Path.read_bytes
    monkeypatch.setattr(Path, "read_bytes", lambda p: read.append(p.name) or read_bytes(p))
    source = [tmp_path / "k.cu"]
    first = build._digest(source, ["-O3"])
    assert first == hashlib.sha256(b"a.cuhoneb.htwok.cukernel-O3").hexdigest()[:16]
    assert build._digest(source, ["-O3"]) == first and build._digest(source, ["-O2"]) != first
    assert sorted(read) == ["a.cuh", "b.h", "k.cu", "k.cu", "k.cu"]
    (tmp_path / "b.h").write_text("three")
    changed = build._digest(source, ["-O3"])
    assert changed != first
    (tmp_path / "b.h").write_text("other")       # of the same size, at another time
    os.utime(tmp_path / "b.h", ns=(1, 1))
    assert build._digest(source, ["-O3"]) not in (first, changed)
    (tmp_path / "c.cuh").write_text("")
    assert build._digest(source, ["-O3"]) == hashlib.sha256(b"a.cuhoneb.hotherc.cuhk.cukernel-O3").hexdigest()[:16]
