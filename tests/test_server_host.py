"""The render server's threads on the CPU, over stand-ins for the device: a server
whose threads cannot all be started is not created and leaves nothing behind, and
requests queued behind one another get each its own frame."""
import subprocess
from pathlib import Path

import pytest

from stratum_hyperdetail_b200.build import host_cxx

ROOT = Path(__file__).resolve().parents[1]
CUDA = Path("/usr/local/cuda/include")


@pytest.fixture(scope="module")
def server(tmp_path_factory):
    if not (CUDA / "cuda_runtime.h").exists():
        pytest.skip("CUDA headers not available")
    exe = tmp_path_factory.mktemp("server") / "server"
    subprocess.run([host_cxx(), "-std=c++17", "-O1", "-I", str(CUDA), str(ROOT / "tests" / "host_server.cpp"),
                    str(ROOT / "stratum_hyperdetail_b200" / "csrc" / "server.cpp"), "-o", str(exe), "-rdynamic", "-pthread",
                    "-ldl"], check=True)
    return lambda *args: subprocess.run([str(exe), *map(str, args)], capture_output=True, text=True, timeout=120)


@pytest.mark.parametrize("started", range(6))
def test_a_thread_that_cannot_be_started(server, started):
    r = server("threads", started)
    assert r.returncode == 0, (r.returncode, r.stdout, r.stderr)


@pytest.mark.parametrize("w,h", [(1, 1), (512, 512), (513, 512), (700, 701)])
def test_queued_requests_get_their_own_frames(server, w, h):
    r = server("frames", w, h)
    assert r.returncode == 0, (r.returncode, r.stdout, r.stderr)
