"""A search context whose creation fails at any of its CUDA calls gives back what it had made: device memory, pinned memory, its stream
and its charge. The library's host code runs on a fake of the CUDA runtime; no GPU is needed."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def exe(vtg_lib, tmp_path_factory):
    out = str(tmp_path_factory.mktemp("faults") / "search_create_faults")
    obj = os.path.join(os.path.dirname(vtg_lib.__file__), "_build", "api_ncc.o")
    subprocess.run(["g++", "-std=c++17", "-O1", "-I" + os.path.join(ROOT, "include"), "-I/usr/local/cuda/include",
                    os.path.join(ROOT, "tests", "c", "search_create_faults.cpp"), obj, "-o", out], check=True, capture_output=True, text=True)
    return out


@pytest.mark.parametrize("call", [None, "cudaSetDevice", "cudaMalloc", "cudaStreamCreateWithFlags", "cudaMemsetAsync",
                                  "cudaStreamSynchronize", "cudaHostAlloc", "cudaHostGetDevicePointer"])
def test_a_failed_creation_leaves_nothing(exe, vtg_lib, call):
    r = subprocess.run([exe] + ([call] if call else []), capture_output=True, text=True, check=True)
    rc, mem, pinned, streams, charge = map(int, r.stdout.split())
    assert (mem, pinned, streams, charge) == (0, 0, 0, 0)
    assert rc == (vtg_lib.OK if call is None else vtg_lib.ENOMEM if call in ("cudaSetDevice", "cudaMalloc") else vtg_lib.ECUDA)
