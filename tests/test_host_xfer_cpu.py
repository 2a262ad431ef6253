"""The host transfer ring's paths without a GPU: csrc/host_xfer.cpp compiled
against a stand-in for the CUDA runtime (xfer_stub.cpp), one process a mode."""
import os
import subprocess

import pytest

from conftest import PKG, ROOT

CUDA = os.environ.get("CUDA_HOME", "/usr/local/cuda")


@pytest.fixture(scope="module")
def stub(tmp_path_factory):
    exe = tmp_path_factory.mktemp("xfer") / "xfer_stub"
    subprocess.run(["g++", "-O1", "-g", "-std=c++17", "-DXFER_IDLE_SECONDS=1", f"-I{CUDA}/include",
                    os.path.join(ROOT, "tests", "xfer_stub.cpp"),
                    os.path.join(PKG, "csrc", "host_xfer.cpp"), "-lpthread", "-o", str(exe)],
                   check=True)
    return str(exe)


def run(stub, mode, limit=60):
    r = subprocess.run([stub, mode], capture_output=True, text=True, timeout=limit)
    assert r.returncode == 0, (mode, r.returncode, r.stderr)


def test_rows_and_their_pads(stub):
    """Rows arrive, the pads of the device's rows are zero (one row and rows longer
    than a slot among them), nothing else is written."""
    run(stub, "copies")


def test_per_thread_stream(stub):
    """No transfer of a copy on cudaStreamPerThread is issued by another thread."""
    run(stub, "per_thread")


@pytest.mark.parametrize("mode", ["fork", "fork_idle"])
def test_forked_child_exits(stub, mode):
    """A child forked with the ring set up (or given back) copies and exits."""
    run(stub, mode)


@pytest.mark.parametrize("mode", ["contexts", "reset_idle"])
def test_contexts(stub, mode):
    """After a reset of the device, and in a context of the program's own, nothing
    touches slots and events of the ring's former context."""
    run(stub, mode)


def test_capture_of_another_thread(stub):
    """Setting the ring up and giving it back leave another thread's capture alone."""
    run(stub, "capture")


def test_results_into_wider_rows(stub):
    """Dense results go into rows with a pitch of their own without the driver's
    copy row by row."""
    run(stub, "pitched_results")
