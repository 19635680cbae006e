"""How the persistent kernels deal their work to CTAs (qmd-progress_b200/csrc/work_lists.h),
compiled for the host: every tile and k-block exactly once, and every piece of a cut tile
found by the CTA that finishes it (CPU, no GPU)."""
import ctypes as C
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "qmd-progress_b200", "csrc")
CUDA_INC = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "include")


@pytest.fixture(scope="module")
def lists(tmp_path_factory):
    cxx = shutil.which("g++") or shutil.which("c++")
    if cxx is None or not os.path.isdir(CUDA_INC):
        pytest.skip("host C++ compiler or CUDA headers not available")
    out = str(tmp_path_factory.mktemp("lists") / "liblists.so")
    subprocess.run([cxx, "-O2", "-std=c++17", "-shared", "-fPIC", "-I" + CUDA_INC, "-I" + CSRC,
                    os.path.join(HERE, "work_lists_harness.cpp"), "-o", out], check=True)
    return C.CDLL(out)


@pytest.mark.parametrize("sms", [148, 132, 7, 1])
@pytest.mark.parametrize("resp", [0, 1])
def test_fp64_shares(lists, sms, resp):
    # every size up to 1300 with the edge of its rule and the next one up, then a few large ones
    for n in list(range(1, 1300)) + [2000, 3500, 4097, 8192, 20011, 32768, 65536]:
        for bt in ((32,) if n <= 416 else (64, 128)):
            assert lists.check_f64(n, bt, resp, sms) == 0, (n, bt)


@pytest.mark.parametrize("sms", [148, 132, 7])
def test_fp64_workspace_covers_every_launch(lists, sms):
    for n in list(range(1, 1300)) + [2000, 4097, 8192, 20011]:
        for resp in (0, 1):
            assert lists.check_f64_workspace(n, resp, sms) == 0, (n, resp)


def test_fp64_launches_stay_short(lists):
    lists.f64_launch_ms.restype = C.c_double
    for n in list(range(1, 1300)) + [2000, 4097, 8192, 12000]:
        for resp in (0, 1):
            assert lists.f64_launch_ms(n, resp) <= 110.0, (n, resp)


@pytest.mark.parametrize("sms", [148, 20])
def test_int8_product_lists(lists, sms):
    for nb in list(range(1, 40)) + [64, 65, 97]:
        assert lists.check_oz(nb, 9, sms) == 0, nb


def test_pair_tile_lists(lists):
    for nb in range(1, 33):
        np2 = (nb + 1) // 2
        count = nb * np2 - np2 * (np2 - 1)
        for whole in {0, 1, count // 2, count}:
            if whole <= count:
                assert lists.check_pair(nb, whole, 1) == 0, (nb, whole)
        assert lists.check_pair(nb, 0, 0) == 0
