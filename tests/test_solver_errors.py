"""The device Newton's host code on a CUDA runtime without a GPU (fake_cuda/):
a call that the runtime refuses leaves nothing running on memory and streams
that go back to their pools, and nothing half made for the next step; what is
timed once is timed once."""
import subprocess
import sys
from pathlib import Path

import pytest

from tdycore_gb300 import build

HERE = Path(__file__).resolve().parent / "fake_cuda"


@pytest.fixture(scope="module")
def fake_library(tmp_path_factory):
    out = tmp_path_factory.mktemp("fake") / "libfake.so"
    include = Path(build._nvcc()).resolve().parents[1] / "include"
    subprocess.run(["g++", "-O1", "-shared", "-fPIC", "-I", str(include), "-o", str(out), str(HERE / "fake_cudart.cpp"),
                    *(str(build.LIBDIR / "obj" / (s + ".o")) for s in build.SOURCES)], check=True)
    return out


def run(library, *args):
    r = subprocess.run([sys.executable, str(HERE / "driver.py"), str(library), *args], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-2000:]


@pytest.mark.parametrize("stream", ["own", "caller"])
def test_refused_calls(fake_library, stream):
    run(fake_library, "refusals", stream)


def test_step_after_a_refused_one(fake_library):
    run(fake_library, "again")


@pytest.mark.parametrize("first", ["fp32", "fp64"])
def test_schedule_is_timed_for_each_precision(fake_library, first):
    run(fake_library, "tuning", first)
