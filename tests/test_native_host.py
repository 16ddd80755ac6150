"""Host code of the library that talks to the CUDA runtime, run on the CPU over a stand-in for that
runtime (tests/native/cuda_runtime.h) whose streams run their work as late as they may."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


def _compiled(tmp_path_factory, name):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("no C++ compiler")
    exe = str(tmp_path_factory.mktemp("native") / name)
    subprocess.run([cxx, "-std=c++17", "-O1", "-g", "-pthread", "-I", os.path.join(HERE, "native"), "-o", exe,
                    os.path.join(HERE, "native", name + ".cc")], check=True)
    return exe


@pytest.fixture(scope="module")
def host_io(tmp_path_factory):
    return _compiled(tmp_path_factory, "host_io_check")


@pytest.mark.parametrize("check", ["arrived unwaited", "arrived waited"])
def test_transfers(host_io, check):
    done = subprocess.run([host_io, check], capture_output=True, text=True, timeout=60)
    assert done.returncode == 0, done.stderr
