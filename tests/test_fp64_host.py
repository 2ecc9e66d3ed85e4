"""CPU checks of the FP64 path's short forms (awfl_pow.cuh, awfl_div.cuh, awfl_device.cuh),
compiled for the host with g++: each equals the general routine it stands in for bit for
bit -- the pressure's pow, the quotients, the WENO reconstruction -- at the edges of its
range and for the values that fall back to the general routine; and the reconstruction's
reverse in stencil differences (awfl_adj.h) equals the general one up to rounding, as does the
FP32 form's reconstruction (awfl_weno32.h)."""
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


def test_short_forms_equal_general_routines(tmp_path):
    exe = str(tmp_path / "fp64_check")
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-mfma", "-I" + CSRC, "-I" + HERE,
                    "-I" + CUDA_INC, os.path.join(HERE, "fp64_host_check.cpp"), "-o", exe], check=True)
    paths = []
    for o in (5, 9):
        t = capi.Context(16, 12, 8, ord_=o, device=-1).tables()
        paths.append(str(tmp_path / ("tables%d.bin" % o)))
        np.concatenate([t["weno_recon"], t["coefs_to_gll"], t["sten_to_gll"], t["deriv"], t["idl"], t["sigma"],
                        t["gll_wts_ngll"]]).astype("<f8").tofile(paths[-1])
    r = subprocess.run([exe] + paths, capture_output=True, text=True)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stdout + r.stderr
