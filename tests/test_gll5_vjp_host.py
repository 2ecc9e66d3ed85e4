"""CPU check, compiled with g++: the adjoint's ord-5 WENO reverse in stencil differences
(awfl_adj.h) is the general one's derivative for stencils of any size."""
import os
import shutil
import subprocess

import numpy as np
import pytest

from awflcloud_b200 import capi

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "awflcloud_b200", "csrc")
CUDA_INC = "/usr/local/cuda/include"

pytestmark = pytest.mark.skipif(shutil.which("g++") is None or not os.path.isdir(CUDA_INC),
                                reason="needs g++ and the CUDA headers")


def test_reverse_equals_the_general_one_at_every_scale(tmp_path):
    exe, tab = str(tmp_path / "check"), str(tmp_path / "tables5.bin")
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-mfma", "-I" + CSRC, "-I" + HERE,
                    "-I" + CUDA_INC, os.path.join(HERE, "gll5_vjp_host_check.cpp"), "-o", exe], check=True)
    t = capi.Context(16, 12, 8, device=-1).tables()
    np.concatenate([t["weno_recon"], t["coefs_to_gll"], t["sten_to_gll"], t["deriv"], t["idl"],
                    t["sigma"]]).astype("<f8").tofile(tab)
    r = subprocess.run([exe, tab], capture_output=True, text=True)
    assert r.stdout.strip() == "ok", r.stdout + r.stderr
