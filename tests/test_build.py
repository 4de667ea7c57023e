"""The build: what makes it run again, and flags whose device code does not depend on the machine."""
import os

import __graft_entry__ as entry


def test_library_is_rebuilt_when_the_flags_change(tmp_path, monkeypatch):
    lib, runs = tmp_path / "libfuelq.so", []

    def compiler(cmd, **_):
        runs.append(cmd)
        lib.write_bytes(b"")

    monkeypatch.setattr(entry, "LIB", str(lib))
    monkeypatch.setattr(entry, "BUILT_WITH", str(tmp_path / "flags"))
    monkeypatch.setattr(entry, "_nvcc", lambda: "nvcc")
    monkeypatch.setattr(entry.subprocess, "run", compiler)
    entry.build_cuda()
    entry.build_cuda()
    assert len(runs) == 1
    monkeypatch.setattr(entry, "NVCC_FLAGS", entry.NVCC_FLAGS + ["-DX"])
    entry.build_cuda()
    assert len(runs) == 2 and "-DX" in runs[1]
    entry.build_cuda()
    assert len(runs) == 2
    os.remove(tmp_path / "flags")   # a library of unknown flags
    entry.build_cuda()
    assert len(runs) == 3


def test_flags_do_not_split_a_module_by_chance():
    assert not any("split-compile" in f for f in entry.NVCC_FLAGS)
