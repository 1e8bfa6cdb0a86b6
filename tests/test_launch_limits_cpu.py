"""Launch limits of the encoder's products, on a preloaded stand-in for the CUDA runtime (fake_cudart.cpp): the
dynamic shared memory that a kernel may take is a property of the device, so a process that uses a second GPU has to be
allowed it there too.  Nothing runs on a GPU."""
import json
import os
import shutil
import subprocess
import sys
from pathlib import Path

import pytest

HERE = Path(__file__).resolve().parent
LIB = HERE.parent / "openadmixture.jl_b200" / "lib" / "libadmix.so"

PROGRAM = r"""
import ctypes as C, json, sys
fake, lib = C.CDLL(sys.argv[1]), C.CDLL(sys.argv[2])
class Net(C.Structure):
    _fields_ = [(n, C.c_int32) for n in ("S", "R", "H", "K")] + [(n, C.c_void_p) for n in ("w1", "b1", "w2", "b2", "w3", "b3")]
class Grads(C.Structure):
    _fields_ = [(n, C.c_void_p) for n in ("w1", "b1", "w2", "b2", "w3", "b3")]
at = C.c_void_p(256)                                   # never read: nothing runs
net, grads = Net(4096, 32, 256, 8, *[256] * 6), Grads(*[256] * 6)
def step(n, device, sms):
    fake.fake_use(device, sms)
    f = lib.admix_mlp_forward(C.byref(net), C.c_int64(n), *[at] * 7, None)
    b = lib.admix_mlp_backward(C.byref(net), C.byref(grads), C.c_int64(n), *[at] * 12, None)
    return {"rc": [f, b], "refused": fake.fake_refused(),
            "cluster": [fake.fake_cluster(i) for i in range(fake.fake_launches())]}
print(json.dumps([step(*job) for job in json.loads(sys.argv[3])]))
"""


@pytest.fixture(scope="module")
def steps(tmp_path_factory):
    cxx, nvcc = shutil.which("g++"), shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    inc = Path(nvcc).resolve().parent.parent / "include"
    if cxx is None or not (inc / "cuda_runtime_api.h").exists():
        pytest.skip("no host compiler or no CUDA headers")
    so = tmp_path_factory.mktemp("fake") / "fake_cudart.so"
    subprocess.run([cxx, "-std=c++17", "-O1", "-shared", "-fPIC", f"-I{inc}", str(HERE / "fake_cudart.cpp"), "-o", str(so)],
                   check=True, capture_output=True)

    def run(*jobs):
        env = dict(os.environ, LD_PRELOAD=str(so))
        r = subprocess.run([sys.executable, "-c", PROGRAM, str(so), str(LIB), json.dumps(jobs)], env=env, capture_output=True,
                           text=True, timeout=120)
        assert r.returncode == 0, r.stderr
        return json.loads(r.stdout)

    return run


def test_a_second_device_is_allowed_the_products_shared_memory(steps):
    for n in (300, 2048, 20000):                          # eight, two and one CTA per tile in the first layer
        for s in steps([n, 0, 148], [n, 1, 148], [n, 0, 148]):
            assert s["rc"] == [0, 0] and s["refused"] == 0, (n, s)


def _first_layer(n, sms):
    """CTAs per tile of the forward pass's first layer: 4 column tiles and 33 blocks of the reduction"""
    tiles = 4 * -(-n // 128)
    return 8 if 6 * tiles <= sms else 2 if 2 * tiles <= sms else 1


def test_tiles_are_shared_by_the_devices_size(steps):
    ns = (1, 128, 300, 768, 769, 1024, 2304, 2305, 4096)
    assert [_first_layer(n, 148) for n in ns] == [8, 8, 8, 8, 2, 2, 2, 1, 1]
    for sms in (148, 74, 296):
        for n, s in zip(ns, steps(*[[n, 0, sms] for n in ns])):
            assert s["rc"] == [0, 0] and s["cluster"][0] == _first_layer(n, sms), (n, sms)
