"""Growth of the context's device buffers against a host-side allocator that
refuses: a refused growth keeps the block in use, an outgrown block is kept for
captured graphs, and the kept blocks stay bounded."""
import shutil
import subprocess
from pathlib import Path

import pytest

HERE = Path(__file__).resolve().parent
CUDA = Path("/usr/local/cuda/include")


@pytest.mark.skipif(shutil.which("g++") is None or not CUDA.exists(), reason="needs g++ and the CUDA headers")
def test_device_buffer_growth(tmp_path):
    exe = tmp_path / "devbuf_host"
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", str(CUDA), "-I", str(HERE.parent / "include"),
                    str(HERE / "cpp" / "devbuf_host.cpp"), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
