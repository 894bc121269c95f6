"""Host paths of the library that need no device (tests/host_paths_driver.cpp)."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def driver(tmp_path_factory):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    cuda = os.path.dirname(os.path.dirname(os.path.realpath(nvcc)))
    lib = os.path.join(cuda, "lib64")
    csrc = os.path.join(ROOT, "dada2-rs_b200", "csrc")
    exe = str(tmp_path_factory.mktemp("hostpaths") / "driver")
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", csrc, "-I", os.path.join(ROOT, "include"), "-I",
                    os.path.join(cuda, "include"), os.path.join(ROOT, "tests", "host_paths_driver.cpp"),
                    os.path.join(csrc, "dgpu_errfun.cpp"), os.path.join(csrc, "dgpu_errfun_external.cpp"), "-o", exe,
                    "-L", lib, f"-Wl,-rpath,{lib}", "-lcudart", "-lpthread"], check=True, capture_output=True)
    return exe


def run(driver, what):
    r = subprocess.run([driver, what], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stdout + r.stderr


def test_scratch_of_the_resident_warps_is_bounded_by_the_tuning(driver):
    run(driver, "geometry")


def test_direct_calls_are_sized_by_the_launch(driver):
    run(driver, "direct_room")


def test_map_call_survives_a_failed_allocation(driver):
    run(driver, "compare_without_memory")
