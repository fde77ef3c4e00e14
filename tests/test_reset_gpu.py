"""The stateless calls after cudaDeviceReset: a program that resets its context and makes new
buffers gets the same answers from them as before. Each call runs in a process of its own."""
import subprocess
import sys

import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu

PROGRAM = """
import ctypes, sys
sys.path.insert(0, {package!r})
import numpy as np
import gsn

n = 3000
rng = np.random.default_rng(1)
keys = rng.integers(0, 2 ** 32, n, dtype=np.uint64).astype(np.uint32)
params = rng.normal(size=(58, n)).astype(np.float32)
image, target = rng.random((48, 64, 3)).astype(np.float32), np.full((48, 64, 3), 70, np.uint8)


def upload(array):
    ptr = gsn.device_alloc(array.nbytes)
    gsn.memcpy(ptr, array.ctypes.data, array.nbytes)
    return ptr


def sort():
    size = gsn.sort_pairs_workspace(n)
    pairs = [upload(keys), upload(np.arange(n, dtype=np.uint32)), upload(keys), upload(keys)]
    status, alt = gsn.sort_pairs(*pairs, n, 0, 32, gsn.device_alloc(size), size)
    assert status == 0, status
    out = np.zeros(n, np.uint32)
    gsn.memcpy(out.ctypes.data, pairs[3 if alt else 1], out.nbytes)
    assert np.array_equal(out, np.argsort(keys, kind="stable"))
    return out.tobytes()


def order():
    perm = upload(keys)
    gsn.spatial_permutation(upload(params), n, perm)
    out = np.zeros(n, np.uint32)
    gsn.memcpy(out.ctypes.data, perm, out.nbytes)
    assert np.array_equal(np.sort(out), np.arange(n))
    return out.tobytes()


def evaluate():
    return gsn.eval_metrics(upload(image), upload(target), 64, 48)


runtime = ctypes.CDLL("/usr/local/cuda/lib64/libcudart.so")
first = {call}()
for _ in range(2):
    assert runtime.cudaDeviceReset() == 0
    assert {call}() == first
"""


@pytest.mark.parametrize("call", ["sort", "order", "evaluate"])
def test_stateless_calls_answer_after_a_reset(call):
    program = PROGRAM.format(package=ROOT + "/gs-native_b200", call=call)
    done = subprocess.run([sys.executable, "-c", program], capture_output=True, text=True, timeout=120)
    assert done.returncode == 0, done.stderr[-2000:]
