"""The switch between the two builds of the library, as the sources read it."""
import os
import subprocess

import pytest

from conftest import REPO

CSRC = os.path.join(REPO, "shallowwaters.jl_b200", "csrc")
CUDA = os.environ.get("CUDA_HOME", "/usr/local/cuda")


@pytest.mark.parametrize("kind", [None, "0", "1"])
def test_packed_products_contract_in_the_fast_build_only(kind):
    """SWB_FAST_BUILD defined as 0 (as the library's sources do) is the parity
    build: a product that feeds a sum is rounded there, as an fma with -0.0."""
    r = subprocess.run(["g++", "-E", "-P", "-x", "c++", f"-I{CUDA}/include", f"-I{REPO}/include"] +
                       ([f"-DSWB_FAST_BUILD={kind}"] if kind else []) + [os.path.join(CSRC, "sw_pack.cuh")],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-2000:]
    assert ("fma.rn.f32x2" in r.stdout) == (kind != "1")
