"""The branch-free quotient and logarithm of the float nodal dS equal CUDA's
correctly rounded division and the scalar logarithm: the logarithm on every
float that it may get, the quotient for every numerator against the
denominators at the edges of the binade, around sqrt(2) and on a few thousand
others, and both over the counts and degrees of a solve.  (All 2^46 pairs of
mantissas: float_terms_main quot 0 8388608, a minute: no
difference.)"""
import os
import shutil
import subprocess

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def differences(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("float_terms") / "float_terms_main")
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    subprocess.run([nvcc, "-O3", "-std=c++17", "-gencode", "arch=compute_100a,code=sm_100a", "-fmad=false", "-I",
                    os.path.join(ROOT, "usap_b200", "csrc"),
                    os.path.join(ROOT, "tests", "float_terms", "float_terms_main.cu"), "-o", exe], check=True)

    def run(*args):
        r = subprocess.run([exe, *map(str, args)], capture_output=True, text=True, timeout=120)
        assert r.returncode == 0, r.stdout + r.stderr
        return int(r.stdout)
    return run


def test_log_equals_scalar_log(differences):
    assert differences("log") == 0


def test_quotient_is_correctly_rounded(differences):
    edges = [(0, 1024), ((1 << 23) - 1024, 1024), (0x3504F3 - 512, 1024), ((1 << 22) - 512, 1024)]
    others = [(lo, 64) for lo in np.random.default_rng(1).integers(0, (1 << 23) - 64, 32)]
    assert differences("quot", *(x for slice_ in edges + others for x in slice_)) == 0


@pytest.mark.parametrize("seed", [1, 2])
def test_terms_over_counts_and_degrees(differences, seed):
    assert differences("range", seed) == 0
