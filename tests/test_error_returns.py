"""Calls that fail half-way and scenes that go while a batch reads them, on the library's own host code over a stand-in for the CUDA runtime (tests/cpp/
fake_cuda.cpp; no GPU): buffers of the device's pool are only freed once nothing queued uses them."""
import os
import subprocess

import pytest

from mobileraytracer_b200 import build as B

HERE = os.path.dirname(os.path.abspath(__file__))
SOURCES = ["mrt_capi.cu", "mrt_bvh.cu", "mrt_grid.cu", "mrt_kernels.cu", "mrt_batch.cu"]


@pytest.fixture(scope="module")
def objects(tmp_path_factory):
    """The library's objects (device code unoptimised: it does not run) and the stand-in's."""
    out = tmp_path_factory.mktemp("objs")
    flags = [f for f in B.NVCC_FLAGS if f not in ("-O3", "-lineinfo")] + ["-Xptxas", "-O0"]
    jobs = []
    for src in SOURCES:
        obj = str(out / src.replace(".cu", ".o"))
        jobs.append((obj, subprocess.Popen([B.NVCC, *flags, "-c", os.path.join(B.CSRC, src), "-o", obj])))
    cuda = os.path.join(os.path.dirname(os.path.dirname(B.NVCC)), "include")
    gxx = ["/usr/bin/g++", "-std=c++17", "-O1", "-g", "-I", cuda]
    fake = str(out / "fake_cuda.o")
    subprocess.run([*gxx, "-c", os.path.join(HERE, "cpp", "fake_cuda.cpp"), "-o", fake], check=True)
    for _, p in jobs:
        assert p.wait() == 0
    return gxx, [o for o, _ in jobs] + [fake], out


def _run(objects, name):
    gxx, objs, out = objects
    exe = str(out / name)
    subprocess.run([*gxx, os.path.join(HERE, "cpp", name + ".cpp"), *objs, "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stdout[-3000:] + r.stderr[-1000:]


def test_scene_creation_and_builds_that_fail(objects):
    _run(objects, "error_returns")


def test_scenes_that_go_while_a_batch_reads_them(objects):
    _run(objects, "scene_in_use")


def test_the_pool_keeps_at_most_a_gibibyte(objects):
    _run(objects, "pool_bound")
