"""CPU checks of the FP32 form's WENO reconstruction (awfl_weno32.h), compiled for the host with
g++, against the general routine in FP64: over the range of values that a field can have (a
tracer's unit is the caller's, so number concentrations of 1e5 and more are ordinary)."""
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


@pytest.fixture(scope="module")
def check(tmp_path_factory):
    d = tmp_path_factory.mktemp("weno32")
    exe = str(d / "check")
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-mfma", "-I" + CSRC, "-I" + HERE,
                    "-I" + CUDA_INC, os.path.join(HERE, "weno32_host_check.cpp"), "-o", exe], check=True)
    paths = []
    for o in (5, 9):
        t = capi.Context(16, 12, 8, ord_=o, device=-1).tables()
        paths.append(str(d / ("tables%d.bin" % o)))
        np.concatenate([t["weno_recon"], t["coefs_to_gll"], t["sten_to_gll"], t["deriv"], t["idl"], t["sigma"],
                        t["gll_wts_ngll"]]).astype("<f8").tofile(paths[-1])

    def run(what):
        r = subprocess.run([exe, what] + paths, capture_output=True, text=True)
        assert r.returncode == 0 and r.stdout.strip() == "ok", r.stdout + r.stderr
    return run


@pytest.mark.parametrize("ord_", [5, 9])
def test_reconstruction_follows_fp64_at_every_scale(check, ord_):
    check("scales%d" % ord_)


@pytest.mark.parametrize("ord_", [5, 9])
def test_errors_no_larger_than_the_matrix_form(check, ord_):
    check("errors%d" % ord_)
