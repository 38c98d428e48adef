"""Failed device allocations inside the C ABI, on the CPU: the entry points'
host code against a stand-in for the CUDA runtime and the kernel launchers
(tests/cpp/alloc_main.cpp), which fails every allocation in turn and checks
every buffer that a launcher is handed afterwards."""
import os
import subprocess

import pytest

from conftest import ROOT
from shapeextraction_b200 import build


@pytest.fixture(scope="module")
def harness(tmp_path_factory):
    tmp = tmp_path_factory.mktemp("alloc")
    flags = ["-O1", "-std=c++17", *build.ARCH, "-ccbin", build._host_cc(), "-I", build.INCLUDE, "-I", build.CSRC]
    jobs = []
    for src in ("capi.cu", "capi_mlp.cu", "capi_batch.cu"):
        obj = str(tmp / (src + ".o"))
        jobs.append((obj, subprocess.Popen([build._nvcc(), *flags, "-c", os.path.join(build.CSRC, src), "-o", obj])))
    main = str(tmp / "main.o")
    jobs.append((main, subprocess.Popen([build._nvcc(), *flags, "-x", "cu", "-c",
                                         os.path.join(ROOT, "tests", "cpp", "alloc_main.cpp"), "-o", main])))
    assert all([p.wait() == 0 for _, p in jobs])
    exe = str(tmp / "alloc_main")
    cuda = os.path.join(os.path.dirname(os.path.dirname(build._nvcc())), "include")
    subprocess.run([build._host_cc(), "-std=c++17", "-I", cuda, os.path.join(ROOT, "tests", "cpp", "alloc_runtime.cpp"),
                    *[o for o, _ in jobs], "-ldl", "-o", exe], check=True)
    return exe


@pytest.mark.parametrize("scenario", ["train", "batch slices", "batch lanes", "queries", "learned", "model",
                                      "foreign"])
def test_a_failed_allocation_leaves_the_context_usable(harness, scenario):
    r = subprocess.run([harness, scenario], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr


def test_the_batch_tuner_times_no_schedule_twice(harness):
    r = subprocess.run([harness, "tuner"], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr


def test_the_cloud_tuner_times_no_setting_twice():
    from shapeextraction_b200 import autotune

    settings = [(min(bucket, 32), halo) for bucket, halo in autotune.CANDIDATES]
    assert len(set(settings)) == len(settings)
