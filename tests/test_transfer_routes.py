"""Which way frames go between host memory and the GPU, and what the copies do when a call fails: transfer.cu compiled
against a CUDA runtime made of host memory (transfer_fakes.cpp), on the CPU."""
import glob
import os
import re
import subprocess

import pytest

from conftest import ROOT
from mypbr_gb300 import build


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("transfer") / "fakes")
    cuda = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(build.nvcc()))), "include")
    subprocess.run(["g++", "-std=c++17", "-O1", "-pthread", "-I" + cuda, os.path.join(ROOT, "tests", "transfer_fakes.cpp"),
                    "-o", out], check=True)
    return out


def holds(program, *scenario):
    r = subprocess.run([program, *map(str, scenario)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, (r.returncode, r.stderr)


# device: a pointer to device memory where host memory is asked for is an error, not an access
@pytest.mark.parametrize("kind", ["pageable", "pinned", "managed", "device"])
def test_a_frame_is_one_transfer(program, kind):
    holds(program, kind)


# from one host page (64 KiB at most), made by one thread and (from 16 MiB) by four, aligned to nothing
@pytest.mark.parametrize("nbytes,offset", [(65536, 0), (65537, 8), (4 << 20, 70001), (20 << 20, 0), ((20 << 20) + 12345, 70001)])
def test_the_pages_of_a_new_frame_are_made_first(program, nbytes, offset):
    holds(program, "new_frame", nbytes, offset)


@pytest.mark.parametrize("scenario", ["out_of_memory", "release", "large", "words"])
def test_kept_memory_makes_room(program, scenario):
    holds(program, scenario)


def test_every_allocation_can_have_the_kept_memory():
    """cudaMalloc is called in transfer.cu alone; the other sources go through device_malloc, which gives kept memory back."""
    for path in glob.glob(os.path.join(ROOT, "mypbr_gb300", "csrc", "**", "*.c*"), recursive=True):
        if os.path.basename(path) != "transfer.cu":
            with open(path) as f:
                assert not re.search(r"\bcudaMalloc(Async|Managed)?\s*\(", f.read()), path
