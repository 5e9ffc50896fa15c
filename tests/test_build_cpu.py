"""The build of the native library where the extension beside it cannot be built (no CUDA compiler needed)."""
import os

import pytest

from powersgd_b200.csrc import build


@pytest.mark.parametrize("stale", [False, True])
def test_without_a_host_compiler_the_library_is_built_all_the_same(stale, tmp_path, monkeypatch):
    nvcc = tmp_path / "nvcc"
    nvcc.write_text('#!/bin/sh\nwhile [ "$1" != "-o" ]; do shift; done\ntouch "$2"\n')
    nvcc.chmod(0o755)
    for name in ("OBJ_DIR", "LIB", "SCAN_LIB"):
        monkeypatch.setattr(build, name, str(tmp_path / name))
    if stale:
        open(build.SCAN_LIB, "w").close()
    monkeypatch.setenv("NVCC", str(nvcc))
    monkeypatch.setenv("CXX", str(tmp_path / "no such compiler"))
    with pytest.warns(UserWarning, match="list checks not built"):
        assert build.build() == build.LIB
    assert os.path.exists(build.LIB) and not os.path.exists(build.SCAN_LIB)
