"""Failure paths of the library's host code, without a GPU: the library's own
objects linked to a stand-in CUDA runtime (tests/cxx/fake_cudart.cpp) in which
device memory is host memory, launches are recorded, and a call can be told to
fail.  Each case of tests/cxx/host_faults.cpp runs as a process of its own.

  host_arrays   calls on host arrays allocate nothing after ap_create, and read no
                array whose copy may still be on its way
  create_fails  ap_create gives back what it took, whichever allocation fails
  tensor_cores_retry  so does the tensor-core solve made on first use, and the next call
                makes all of it
  solver_info   ap_solver_info reports a tensor-core path that cannot be made as
                unavailable, and does not change the handle's solver
  device_output  a device pointer given for a host output is refused by the copy, not
                written by the host
  shared_memory_limits  a batch of small grids leaves a batch of large ones its
                kernel's shared memory
  trial_graphs  the loop runs on one trial a graph launch where the graph of four
                cannot be made
  profile_launches  ap_profile_stages launches the kernels that a trial does
  null_stream_waits  what a call copies or clears on the null stream has arrived before
                a launch on a stream of the library's own
  batch_blocks  a batch of few work items launches no more blocks than items
  small_calls   calls on host arrays of a small design wait for the device once
  outputs_in_bounds  the host touches no page outside a result's array
"""
import os
import subprocess

import pytest

from conftest import REPO

CXX = os.path.join(REPO, "tests", "cxx")
CUDA_INC = "/usr/local/cuda/include"


@pytest.fixture(scope="module")
def host_faults(tmp_path_factory):
    from aieplace_gb300 import build

    if not os.path.isdir(CUDA_INC):
        pytest.skip("no CUDA headers")
    build.build()
    objs = [os.path.join(build.BUILD, os.path.splitext(s)[0] + ".o") for s in build.SOURCES]
    if not all(map(os.path.exists, objs)):
        build.build(force=True)
    exe = str(tmp_path_factory.mktemp("host_faults") / "host_faults")
    cmd = ["g++", "-std=c++17", "-O1", "-Wall", "-Werror", "-I", os.path.join(REPO, "include"), "-I", CXX,
           "-isystem", CUDA_INC, os.path.join(CXX, "host_faults.cpp"), os.path.join(CXX, "fake_cudart.cpp"), *objs,
           "-o", exe]
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    return exe


@pytest.mark.parametrize("case", ["host_arrays", "create_fails", "tensor_cores_retry", "solver_info", "device_output",
                                  "shared_memory_limits", "trial_graphs", "profile_launches", "null_stream_waits",
                                  "batch_blocks", "small_calls", "outputs_in_bounds"])
def test_host_faults(host_faults, case):
    r = subprocess.run([host_faults, case], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, f"exit {r.returncode}\n{r.stderr}"
