"""The library's host code without a GPU: nc_api.cu, nc_pool.cu, nc_batch.cu, nc_serve.cu and
nc_noalloc.cu compiled as C++ against a CUDA runtime of host memory (tests/cpp/fake_device.h)."""
import concurrent.futures as cf
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "neurocorrelation_gb300", "csrc")
CUDA_INC = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "include")
SOURCES = [os.path.join(CSRC, f) for f in ("nc_api.cu", "nc_pool.cu", "nc_batch.cu", "nc_serve.cu", "nc_noalloc.cu", "nc_host.cpp")]


@pytest.fixture(scope="module")
def host_paths(tmp_path_factory):
    if not os.path.exists(os.path.join(CUDA_INC, "cuda_runtime.h")):
        pytest.skip("CUDA headers not found")
    tmp = tmp_path_factory.mktemp("host_paths")
    sources = SOURCES + [os.path.join(ROOT, "tests", "cpp", "host_paths.cpp")]
    objs = [str(tmp / (os.path.basename(s) + ".o")) for s in sources]

    def compile_one(pair):
        subprocess.run(["g++", "-std=c++17", "-O1", "-ffp-contract=off", "-I" + CSRC, "-I" + CUDA_INC, "-x", "c++",
                        "-c", pair[0], "-o", pair[1]], check=True)

    with cf.ThreadPoolExecutor(8) as ex:
        list(ex.map(compile_one, zip(sources, objs)))
    exe = str(tmp / "host_paths")
    subprocess.run(["g++", "-o", exe, *objs, "-lpthread"], check=True)
    return exe


@pytest.mark.parametrize("check", ["weights_order", "raster_order", "raster_refused",
                                   "detectors_order", "detectors_refused",
                                   "reads_allocate_nothing", "no_index",
                                   "failed_read", "server_read_fails", "server_device_lost", "footprint",
                                   "row_plan", "flush_then_step"])
def test_host_path(host_paths, check):
    r = subprocess.run([host_paths, check], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout + r.stderr
    assert r.stdout.strip().endswith("OK")
