"""Calls while the device has next to no memory left: what needed only a few bytes of scratch, or had a route
that needs less, still works.  In child processes, so that the memory that other tests leave with the library
plays no part; kernels are loaded beforehand, since loading one needs memory too."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

_PREAMBLE = r"""
import ctypes, sys
sys.path.insert(0, sys.argv[1])
import torch
from cuda.bindings import runtime as rt
from haskell_infer_demo_b200 import lib as L
from haskell_infer_demo_b200 import ops
lib = L.load()
stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)

class Full:
    '''Takes the device's memory until between `leave` and `leave` + 2 MiB are free.'''
    def __init__(self, leave):
        self.leave, self.held = leave, []
    def __enter__(self):
        step = 1 << 36
        while step >= 1 << 21:
            if torch.cuda.mem_get_info()[0] - step >= self.leave:
                err, p = rt.cudaMalloc(step)
                if int(err) == 0:
                    self.held.append(p)
                    continue
                rt.cudaGetLastError()
            step //= 2
        print('free', torch.cuda.mem_get_info()[0])
    def __exit__(self, *exc):
        for p in self.held:
            rt.cudaFree(p)

def message():
    return lib.ffn_int4_last_error().decode()
"""

_QUANTIZER = _PREAMBLE + r"""
n, k = 5120, 17408                                   # 46 MB of bytes
w = torch.empty((n, k), device='cuda').normal_(0.0, 0.02)
packed = torch.full((n, k // 2), 0xAB, dtype=torch.uint8, device='cuda')
scales = torch.full((n, k // 128), 0x1234, dtype=torch.int16, device='cuda')
call = lambda: lib.ffn_quantize_int4(w.data_ptr(), packed.data_ptr(), scales.data_ptr(), n, k, stream)
kept = w[1234, 567].item()
w[1234, 567] = float('nan')
torch.cuda.synchronize()
with Full(8 << 20):
    st = call()
assert st == -3 and str(1234 * k + 567) in message(), (st, message())
assert (packed == 0xAB).all() and (scales == 0x1234).all()         # refused: nothing written
w[1234, 567] = kept
torch.cuda.synchronize()
with Full(8 << 20):
    st = call()
assert st == 0, message()
want_p, want_s = ops.quantize_int4(w)
assert torch.equal(packed, want_p) and torch.equal(scales, want_s.view(torch.int16))
print('quantized')
"""

def child(code):
    proc = subprocess.run([sys.executable, "-c", code, ROOT], capture_output=True, text=True, timeout=600,
                          env=dict(os.environ, CUDA_MODULE_LOADING="EAGER"))
    assert proc.returncode == 0, proc.stdout[-2000:] + proc.stderr[-3000:]
    return proc.stdout


def test_quantizer_needs_a_few_bytes_only(cuda):
    assert "quantized" in child(_QUANTIZER)
