"""Registers of the FP64 operator kernels (krylov.cu compiled for sm_100a at orders 2, 6 and 8, no
GPU), as ptxas reports them. A stated minimum of resident CTAs is a limit that spills at order 8,
and at order 2 an explicit one makes the compiler spend registers (160 for 128) where it has
no use for them. So: nothing spills at order 8; outside the iteration order 2 fits four CTAs
an SM (128 registers) and the operator alone spills nowhere; inside it order 6 keeps three CTAs.
"""

import os
import re
import shutil
import subprocess

import pytest

REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(REPO, "ho-cxx_b200", "csrc")

SOURCE = """
#define HO2D_KSWITCH(K, CALL)                          \\
    switch (K) {                                       \\
        case 2: { constexpr int KK = 2; CALL; } break; \\
        case 6: { constexpr int KK = 6; CALL; } break; \\
        case 8: { constexpr int KK = 8; CALL; } break; \\
        default: return cudaErrorInvalidValue;         \\
    }
#include "krylov.cu"
"""


@pytest.fixture(scope="module")
def kernels(tmp_path_factory):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("nvcc not available")
    d = tmp_path_factory.mktemp("registers")
    (d / "k.cu").write_text(SOURCE)
    r = subprocess.run([nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17", "-I", CSRC, "-I",
                        os.path.join(REPO, "include"), "--expt-relaxed-constexpr", "-Xptxas", "-O3,-v", "-c",
                        str(d / "k.cu"), "-o", str(d / "k.o")], check=True, capture_output=True, text=True)
    out, name, spill = {}, None, 0
    for line in r.stderr.splitlines():
        if m := re.search(r"Compiling entry function '\S*?(k_mf_(?:v|t|init|residual|apply))ILi(\d)Ed", line):
            name = (m.group(1), int(m.group(2)))
        elif "Compiling entry function" in line:
            name = None
        elif m := re.search(r"(\d+) bytes spill stores", line):
            spill = int(m.group(1))
        elif (m := re.search(r"Used (\d+) registers", line)) and name:
            out[name] = (int(m.group(1)), spill)
    return out


def test_order_8_does_not_spill(kernels):
    for k in ("k_mf_v", "k_mf_t", "k_mf_init", "k_mf_residual", "k_mf_apply"):
        assert kernels[k, 8][1] == 0, (k, kernels[k, 8])


def test_order_2_outside_the_iteration_fits_four_ctas(kernels):
    for k in ("k_mf_init", "k_mf_residual", "k_mf_apply"):
        assert kernels[k, 2][0] <= 128 and kernels[k, 2][1] == 0, (k, kernels[k, 2])


def test_order_6(kernels):
    assert kernels["k_mf_apply", 6][1] == 0
    for k in ("k_mf_v", "k_mf_t"):
        assert kernels[k, 6][0] <= 168  # three CTAs of 128 threads in 65,536 registers
