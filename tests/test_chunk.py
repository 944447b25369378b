"""The chunk length of the marching kernels (csrc/nova_chunk.h): the shortest
search gives the rule's answer, and a call costs little beside a launch.  CPU only."""
import os
import subprocess

from conftest import ROOT


def test_distinct_chunks_give_the_rules_answer(tmp_path):
    exe = str(tmp_path / "chunk")
    subprocess.run(["g++", "-std=c++17", "-O2", "-Wall", "-Werror", "-I" + os.path.join(ROOT, "novaclone_b200", "csrc"),
                    os.path.join(ROOT, "tests", "cpp", "chunk_driver.cpp"), "-o", exe], check=True)
    r = subprocess.run([exe, "4096"], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
    ours, every = (float(v) for v in r.stdout.split())
    assert ours < every / 8  # 127 distinct chunks of 4096 counts
