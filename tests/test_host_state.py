"""Host-side state of libgeofd, run against a CUDA runtime without a device
(fake_cuda.h): what belongs to a device is set up on every device, and runs
that do not fit in memory at once."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PKG = os.path.join(ROOT, "geophysics_gb300")


@pytest.fixture(scope="module")
def check(tmp_path_factory):
    cxx = shutil.which("g++") or shutil.which("c++")
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    inc = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(nvcc))), "include")
    lib = os.path.join(PKG, "libgeofd.so")
    if not cxx or not os.path.exists(os.path.join(inc, "cuda_runtime.h")) or not os.path.exists(lib):
        pytest.skip("needs a C++ compiler, the CUDA headers and the built library")
    exe = str(tmp_path_factory.mktemp("host_state") / "host_state_check")
    subprocess.run([cxx, "-O1", "-std=c++17", "-I" + os.path.join(ROOT, "include"),
                    "-I" + os.path.join(PKG, "csrc"), "-I" + inc,
                    os.path.join(ROOT, "tests", "host_state_check.cpp"), "-o", exe, lib, "-rdynamic",
                    "-Wl,-rpath," + PKG, "-Wl,--allow-shlib-undefined", "-lpthread"], check=True)

    def run(name):
        # freed memory is overwritten
        env = dict(os.environ, MALLOC_PERTURB_="165")
        r = subprocess.run([exe, name], capture_output=True, text=True, timeout=300, env=env)
        assert r.returncode == 0, r.stdout[-3000:] + r.stderr[-1000:]
        return r.stdout

    return run


def test_second_device_gets_tables_and_kernel_attributes(check):
    """Every entry point on one device, then on another: the same constant
    tables are copied to both, the same kernels' shared-memory limits set.
    No call waits for the whole device (a graph that another host thread
    captures would fail)."""
    check("devices")


def test_batched_rtm_beyond_memory_runs_in_groups(check):
    check("batch_memory")


def test_2d_rtm_tile_widths(check):
    check("plans")


def test_codec_scratch_that_failed_to_grow(check):
    check("codec_growth")


def test_codec_scratch_is_what_its_kernels_use(check):
    check("codec_memory")


def test_small_batch_spreads_over_the_warps(check):
    check("batch_spread")


def test_detector_scans_before_the_next_lines_go_in(check):
    check("watch_order")


def test_tilted_step_keeps_its_maps(check):
    check("tti_maps")


def test_any_chunk_override_covers_the_windows(check):
    check("batch_chunk_override")
