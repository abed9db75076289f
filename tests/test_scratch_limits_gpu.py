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

_FFN = _PREAMBLE + r"""
h, i = 5120, 17408
gen = torch.Generator(device='cuda').manual_seed(3)
# any bytes are weights; made without the quantizer, whose pool would hold memory that the driver can take back
weights = [(torch.randint(0, 256, (n, k // 2), dtype=torch.uint8, device='cuda', generator=gen),
            (0.002 + 0.002 * torch.rand((n, k // 128), device='cuda', generator=gen)).to(torch.bfloat16)) for n, k in ((2 * i, h), (h, i))]
torch.cuda.synchronize()
torch.cuda.empty_cache()
mlp = ops.DenseMlp(*weights[0], *weights[1])
state = {}
for m in (3, 128):
    x = torch.randn((m, h), device='cuda', generator=gen).to(torch.bfloat16)
    state[m] = x, mlp.workspace(m), torch.empty_like(x)
mlp.forward_mlp_prepared(state[3][0][:1].contiguous())             # the status word
torch.cuda.synchronize()
with Full(20 << 20):                                               # the pairs need 14 MB, 512 tokens' scratch 42
    got = {m: (mlp.forward_mlp_prepared(*state[m]), L.device_status())[0].clone() for m in state}
for m in state:
    want = mlp.forward_mlp_prepared(*state[m])
    L.device_status()
    # another split of the tokens and of K over CTAs: FP32 order, then BF16 roundings of act and y
    err = ((got[m].float() - want.float()).norm() / want.float().norm()).item()
    print(m, 'tokens, relative difference', err)
    assert err <= 2.0 ** -8
print('computed')
"""


def child(code):
    proc = subprocess.run([sys.executable, "-c", code, ROOT], capture_output=True, text=True, timeout=600,
                          env=dict(os.environ, CUDA_MODULE_LOADING="EAGER"))
    assert proc.returncode == 0, proc.stdout[-2000:] + proc.stderr[-3000:]
    return proc.stdout


def test_quantizer_needs_a_few_bytes_only(cuda):
    assert "quantized" in child(_QUANTIZER)


def test_batched_ffn_makes_do_with_what_the_pairs_needed(cuda):
    assert "computed" in child(_FFN)
