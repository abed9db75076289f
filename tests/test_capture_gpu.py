"""A GEMM of three rows and more under stream capture: the graph holds kernels only - so it can be instantiated
more than once, cloned or used as a child - whether or not the device has run such a call before, and a call that
another thread makes meanwhile neither fails nor breaks the capture.  An FFN of 128 tokens after a call of 8 only.
In child processes, since a device's first call is the interesting one."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

_PREAMBLE = r"""
import sys, threading
sys.path.insert(0, sys.argv[1])
import torch
from cuda.bindings import runtime as rt
from haskell_infer_demo_b200 import lib as L
from haskell_infer_demo_b200 import ops
lib = L.load()
n, k, rows = 8192, 2560, 37
gen = torch.Generator(device='cuda').manual_seed(11)
packed, scales = ops.quantize_int4(torch.empty((n, k), device='cuda').normal_(0.0, 0.02, generator=gen))
w = ops.dequantize_int4(packed, scales)[0].double()
a = torch.empty((rows, k), dtype=torch.bfloat16, device='cuda')
out = torch.empty((rows, n), dtype=torch.bfloat16, device='cuda')
def fresh():
    a.copy_(torch.randn((rows, k), device='cuda', generator=gen))
def call(a=a, out=out):
    L.check(lib.ffn_gemm_int4_bf16(a.data_ptr(), packed.data_ptr(), scales.data_ptr(), out.data_ptr(), rows, n, k, 128,
                                   torch.cuda.current_stream().cuda_stream))
def right(a=a, out=out):
    want = a.double() @ w.T
    # half a BF16 ulp, and FP32 sums: 128 products a group, some 20 groups and a few partial sums
    bound = want.abs() * 2.0 ** -8 + (a.double().abs() @ w.abs().T) * (160 * 2.0 ** -24)
    return bool(((out.double() - want).abs() <= bound).all())
def capture(body):
    graph = torch.cuda.CUDAGraph(keep_graph=True)
    with torch.cuda.graph(graph, capture_error_mode='global'):
        body()
    raw = rt.cudaGraph_t(graph.raw_cuda_graph())
    err, nodes, count = rt.cudaGraphGetNodes(raw, 64)
    kinds = [rt.cudaGraphNodeGetType(nodes[i])[1].name for i in range(count)]
    assert kinds and set(kinds) == {'cudaGraphNodeTypeKernel'}, kinds
    for _ in range(2):                                              # a graph with memory nodes refuses the second
        err, _ = rt.cudaGraphInstantiate(raw, 0)
        assert int(err) == 0, err
    graph.instantiate()
    return graph
def replays(graph):
    for _ in range(3):
        fresh()
        out.zero_()
        graph.replay()
        assert right()
torch.cuda.synchronize()
"""

_BEFORE_AND_AFTER = _PREAMBLE + r"""
first = capture(call)                                               # this device has run no such call yet
replays(first)
fresh()
call()
assert right()
later = capture(call)
replays(later)
replays(first)
L.device_status()
print('captured')
"""

_ANOTHER_THREAD = _PREAMBLE + r"""
a2, out2 = torch.randn((rows, k), device='cuda', generator=gen).to(torch.bfloat16), torch.empty_like(out)
side, errors = torch.cuda.Stream(), []
def other():
    try:
        with torch.cuda.stream(side):
            for _ in range(2):                                      # the device's first call, and a later one
                call(a2, out2)
    except Exception as e:
        errors.append(e)
def body():
    t = threading.Thread(target=other)
    t.start()
    t.join()
    call()
torch.cuda.synchronize()
graph = capture(body)
assert not errors, errors
side.synchronize()
assert right(a2, out2)
replays(graph)
L.device_status()
print('captured')
"""

_LONG_FFN_AFTER_A_SHORT_ONE = _PREAMBLE + r"""
h, i = 2560, 2176
mlp = ops.DenseMlp(*[t for s in ((2 * i, h), (h, i)) for t in ops.quantize_int4(torch.empty(s, device='cuda').normal_(0.0, 0.02, generator=gen))])
x = torch.randn((128, h), device='cuda', generator=gen).to(torch.bfloat16)
ws, y = mlp.workspace(128), torch.empty_like(x)
mlp.forward_mlp_prepared(x[:8].contiguous())
torch.cuda.synchronize()
graph = capture(lambda: mlp.forward_mlp_prepared(x, ws, y))
for _ in range(2):
    x.copy_(torch.randn((128, h), device='cuda', generator=gen))
    graph.replay()
    got = y.clone()
    want = mlp.forward_mlp_prepared(x)                              # in one launch, the region for it being had now
    # another split of the tokens and of K over CTAs: FP32 order, then BF16 roundings of act and y
    assert (got.float() - want.float()).norm() / want.float().norm() <= 2.0 ** -8
L.device_status()
print('captured')
"""


@pytest.mark.parametrize("code", [_BEFORE_AND_AFTER, _ANOTHER_THREAD, _LONG_FFN_AFTER_A_SHORT_ONE],
                         ids=["first_and_later_call", "another_threads_call", "long_ffn_after_a_short_one"])
def test_captured_calls(cuda, code):
    proc = subprocess.run([sys.executable, "-c", code, ROOT], capture_output=True, text=True, timeout=600)
    assert proc.returncode == 0 and "captured" in proc.stdout, proc.stdout[-2000:] + proc.stderr[-3000:]
