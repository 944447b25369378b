"""The cache of idle device buffers (csrc/nova_bufcache.h), compiled against a
counted stand-in for cudaFree: no buffer is lost or freed twice.  CPU only."""
import os
import subprocess

import pytest

from conftest import ROOT

CUDA_INC = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "include")


@pytest.fixture(scope="module")
def driver(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("bufcache") / "driver")
    subprocess.run(["g++", "-std=c++17", "-O1", "-Wall", "-Werror", "-pthread", "-I" + CUDA_INC,
                    "-I" + os.path.join(ROOT, "novaclone_b200", "csrc"),
                    os.path.join(ROOT, "tests", "cpp", "bufcache_driver.cpp"), "-o", exe], check=True)
    return exe


# close_race: buffers dropped on other threads while the context is destroyed
# host_memory: no room on the host to note a buffer (an exception must not leave a C entry point)
# out_of_memory: a failed device allocation or FFT plan gets the idle buffers of every context
@pytest.mark.parametrize("scenario", ["bound_and_reuse", "close_race", "host_memory", "out_of_memory"])
def test_every_buffer_is_freed_once(driver, scenario):
    r = subprocess.run([driver, scenario], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout
