"""The helper threads' source builds where the host has no SSE2 (B200 boards come
with Arm hosts too): compiled with the macro undefined and an emmintrin.h that
refuses to be included."""
import shutil
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "oxideav-av1_b200" / "csrc"


@pytest.mark.skipif(not shutil.which("g++"), reason="no g++")
def test_host_pool_builds_without_sse2(tmp_path):
    (tmp_path / "emmintrin.h").write_text("#error no such header on this host\n")
    r = subprocess.run(["g++", "-std=c++17", "-fsyntax-only", "-U__SSE2__", f"-I{tmp_path}", f"-I{CSRC}",
                        str(CSRC / "host_pool.cpp")], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
