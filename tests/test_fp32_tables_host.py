"""CPU check, compiled with g++: an FP32 context is created only if the transform tables hold the
constants that its kernels have as literals (awfl_recip.h)."""
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


def test_fp32_constants_are_compared_with_the_tables(tmp_path):
    exe = str(tmp_path / "check")
    subprocess.run(["g++", "-O1", "-std=c++17", "-I" + CSRC, "-I" + HERE, "-I" + CUDA_INC,
                    os.path.join(HERE, "fp32_tables_host_check.cpp"), "-o", exe], check=True)
    paths = []
    for o in (5, 9):
        t = capi.Context(16, 12, 8, ord_=o, device=-1).tables()
        paths.append(str(tmp_path / ("tables%d.bin" % o)))
        np.concatenate([t["weno_recon"], t["coefs_to_gll"], t["sten_to_gll"], t["deriv"], t["idl"],
                        t["sigma"]]).astype("<f8").tofile(paths[-1])
    r = subprocess.run([exe] + paths, capture_output=True, text=True)
    assert r.stdout.strip() == "done", r.stdout + r.stderr
