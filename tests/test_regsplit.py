"""The register budget of the warp-specialised kernels (csrc/nova_regsplit.h):
setmaxnreg.inc waits without end when the registers a block was launched with
do not cover the split, so the launch is refused then.  CPU only."""
import os
import subprocess

import pytest

from conftest import ROOT

# (registers at launch, consumers, inc, producers, dec): the splits of the FP64 stage, FP64 MHD and adjoint kernels
STAGE, MHD = (512, 112, 128, 24), (256, 232, 128, 24)


@pytest.fixture(scope="module")
def fits(tmp_path_factory):
    d = tmp_path_factory.mktemp("regsplit")
    src = d / "m.cpp"
    src.write_text('#include "nova_regsplit.h"\n#include <cstdlib>\n'
                   "int main(int, char **v) { return nova::reg_split_fits(atoi(v[1]), atoi(v[2]), atoi(v[3]), "
                   "atoi(v[4]), atoi(v[5])) ? 0 : 1; }\n")
    subprocess.run(["g++", "-std=c++17", "-I" + os.path.join(ROOT, "novaclone_b200", "csrc"), str(src), "-o",
                    str(d / "m")], check=True)
    return lambda regs, split: subprocess.run([str(d / "m"), str(regs)] + [str(v) for v in split]).returncode == 0


@pytest.mark.parametrize("regs,split,want", [
    (96, STAGE, True),    # 60416 of 61440
    (93, STAGE, True),    # allocated as 96
    (88, STAGE, False),   # 56320 at launch
    (120, STAGE, False),  # above what the consumers would rise to
    (168, MHD, True),     # 62464 of 64512
    (160, MHD, False),    # 61440 at launch
    (16, STAGE, False),   # below what the producers would fall to
])
def test_budget(fits, regs, split, want):
    assert fits(regs, split) == want
