"""The library is rebuilt when any file that goes into it is newer (no compiler, no GPU)."""
import os

import pytest

from vlasov1d2v_b200 import build


@pytest.mark.parametrize("changed", ["a.cu", "a.cuh", "a.h", "vlasov1d2v.h", None])
def test_needs_build(tmp_path, monkeypatch, changed):
    csrc, include = tmp_path / "csrc", tmp_path / "include"
    csrc.mkdir()
    include.mkdir()
    files = [csrc / "a.cu", csrc / "a.cuh", csrc / "a.h", csrc / "notes.txt", include / "vlasov1d2v.h"]
    lib = tmp_path / "lib.so"
    for f in files + [lib]:
        f.write_text("")
        os.utime(f, (1000, 1000 if f != lib else 2000))
    monkeypatch.setattr(build, "CSRC", str(csrc))
    monkeypatch.setattr(build, "INCLUDE", str(include))
    monkeypatch.setattr(build, "LIB", str(lib))
    for f in files:
        if f.name == changed:
            os.utime(f, (3000, 3000))
    assert build.needs_build() == (changed is not None)
    lib.unlink()
    assert build.needs_build()
