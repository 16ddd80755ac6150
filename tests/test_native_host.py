"""Host code of the library that talks to the CUDA runtime, run on the CPU over a stand-in for that
runtime (tests/native/cuda_runtime.h) whose streams run their work as late as they may."""
import os
import shutil
import subprocess
import sys

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


@pytest.mark.parametrize("check", ["arrived unwaited", "arrived waited", "upload without an event",
                                   "download without an event", "download without a record", "no room for threads"])
def test_transfers(host_io, check):
    done = subprocess.run([host_io, check], capture_output=True, text=True, timeout=20)
    assert done.returncode == 0, done.stderr


@pytest.fixture(scope="module")
def host_rules(tmp_path_factory):
    return _compiled(tmp_path_factory, "host_rules_check")


@pytest.mark.parametrize("check", ["size classes", "slices"])
def test_rules(host_rules, check):
    done = subprocess.run([host_rules, check], capture_output=True, text=True, timeout=20)
    assert done.returncode == 0, done.stderr


@pytest.fixture(scope="module")
def solo_layout(tmp_path_factory):
    return _compiled(tmp_path_factory, "solo_layout_check")


@pytest.mark.parametrize("check", ["stores", "tiles"])
def test_a_warp_per_stream(solo_layout, check):
    done = subprocess.run([solo_layout, check], capture_output=True, text=True, timeout=20)
    assert done.returncode == 0, done.stderr


@pytest.fixture(scope="module")
def encode_layout(tmp_path_factory):
    return _compiled(tmp_path_factory, "encode_layout_check")


@pytest.mark.parametrize("check", ["residents", "buffers", "banks"])
def test_the_encoders_shared_memory(encode_layout, check):
    done = subprocess.run([encode_layout, check], capture_output=True, text=True, timeout=20)
    assert done.returncode == 0, done.stderr


@pytest.fixture(scope="module")
def host_pool(tmp_path_factory):
    return _compiled(tmp_path_factory, "host_pool_check")


@pytest.mark.parametrize("check", ["old sizes make room", "random use"])
def test_result_memory(host_pool, check):
    done = subprocess.run([host_pool, check], capture_output=True, text=True, timeout=20)
    assert done.returncode == 0, done.stderr


def test_no_result_memory_is_an_answer():
    """More than there is, up to what no class could hold: NULL at once."""
    from lmz_b200 import build
    code = ("import ctypes, sys; lib = ctypes.CDLL(sys.argv[1]); f = lib.lmz_gpu_host_alloc; f.restype = ctypes.c_void_p;"
            "f.argtypes = [ctypes.c_size_t]; print([f(n) for n in (1 << 62, (1 << 63) + 1, (1 << 64) - 65, (1 << 64) - 1)])")
    out = subprocess.run([sys.executable, "-c", code, build.build()], capture_output=True, text=True, timeout=60)
    assert out.stdout.strip() == "[None, None, None, None]", out.stderr


def test_a_mapping_that_is_not_written_through_is_given_back(monkeypatch):
    import contextlib

    import torch
    from lmz_b200 import gpu, save
    monkeypatch.setattr(torch.cuda, "device", lambda d: contextlib.nullcontext())
    monkeypatch.setattr(gpu, "last_error", lambda: "made to fail")
    seen = []

    class Lib:
        def lmz_host_map_file(self, fd, off, n):
            return 4096

        def lmz_gpu_transfer_download(self, *a):
            return gpu.ECUDA

        def lmz_host_unmap_file(self, at, n):
            seen.append((at, n))

    class Data:
        def numel(self):
            return 100

        def data_ptr(self):
            return 0

    w = save._FileWriter.__new__(save._FileWriter)
    w.lib, w.fd, w.device, w.stream, w.handle, w.pending = Lib(), 3, None, 0, 1, []
    with pytest.raises(RuntimeError):
        w.send(Data(), 4100)
    assert seen == [(4096, 104)] and not w.pending
