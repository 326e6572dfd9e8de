"""The zstd decoder's workspace is read in the types that it was written in (its host builds run with no
barrier between a batch of stores and the loads that follow)."""
import shutil
import subprocess

import pytest

from test_zstd_host import HARNESS, HEADER


def test_no_type_punned_workspace(tmp_path):
    cxx = shutil.which("g++")
    if not cxx:
        pytest.skip("no host C++ compiler")
    shutil.copy(HEADER, tmp_path / "zstd_dec.cuh")
    (tmp_path / "h.cpp").write_text(HARNESS)
    r = subprocess.run([cxx, "-O2", "-std=c++20", "-Wstrict-aliasing=2", "-Werror", "-c",
                        str(tmp_path / "h.cpp"), "-o", str(tmp_path / "h.o")], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[:3000]
