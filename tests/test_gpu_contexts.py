"""The C entry points after a device reset: what the library keeps per context (shared-memory limits, addresses of its own
variables) has to be made again.  In a process of its own, without torch's tensors."""
import subprocess
import sys
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu

CODE = """
import ctypes
from ctypes import byref, c_char_p, c_size_t, c_void_p
import torch  # loads the CUDA runtime
from kernelfuser_b200 import _lib
rt, lib = ctypes.CDLL('libcudart.so.12'), _lib.load()

def alloc(n):
    p = c_void_p()
    assert rt.cudaMalloc(byref(p), c_size_t(n)) == 0 and rt.cudaMemset(p, 0, c_size_t(n)) == 0
    return p.value

def call(D, variant):
    S = 256
    q, k, v, kn, o, g = (alloc(2 * 2 * S * D) for _ in range(6))
    word, st = alloc(16), [2 * S * D, S * D, D]
    rc = lib.kf_optimized_attention(q, k, v, g, g, None, None, kn, o, 1, 2, 2, S, D, 0, 1, 1, 1e-6, 0.06, *(st * 5), word,
                                    variant, None)
    assert rc == 0, lib.kf_last_error()
    rc = lib.kf_optimized_attention_static(q, k, v, g, g, None, None, o, 1, 2, 2, S, D, 0, 1, 1, 1e-6, 0.06, *(st * 4),
                                           word, None)
    assert rc == 0, lib.kf_last_error()
    assert rt.cudaDeviceSynchronize() == 0
    host = ctypes.c_int(7)
    assert rt.cudaMemcpy(byref(host), c_void_p(word), c_size_t(4), 2) == 0 and host.value == 0

for _ in range(2):
    for D, variants in ((128, (0, 1, 2, 3)), (256, (0, 1, 3))):
        for variant in variants:
            call(D, variant)
    assert rt.cudaDeviceReset() == 0
"""


def test_calls_after_a_device_reset():
    root = Path(__file__).resolve().parent.parent
    r = subprocess.run([sys.executable, "-c", CODE], cwd=root, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
