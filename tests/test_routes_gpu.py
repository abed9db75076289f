"""Which kernel serves a call, by the names of the kernels that run: the tests of results alone would pass on the
kernels that stand behind the intended one, too."""
import pytest
import torch

import gpu_util
from haskell_infer_demo_b200 import lib as L
from haskell_infer_demo_b200 import ops

pytestmark = pytest.mark.gpu


def kernels(call):
    seen = gpu_util.kernels(call)
    if seen is None:
        pytest.skip("the profiler reports no kernels here")
    return seen


def layer(cuda, hidden, inter):
    q = lambda n, k: ops.quantize_int4(torch.empty((n, k), device=cuda).normal_(0.0, 0.02))
    return ops.DenseMlp(*q(2 * inter, hidden), *q(hidden, inter), post_norm_w=torch.zeros(hidden, dtype=torch.bfloat16, device=cuda))


@pytest.mark.parametrize("tokens", [3, 4])
def test_a_prepared_layer_keeps_its_kernel_with_and_without_the_norm(cuda, tokens):
    mlp = layer(cuda, 1024, 3072).prepare()
    x = torch.randn((tokens, 1024), device=cuda).to(torch.bfloat16)
    old = L.load().ffn_int4_set_decode_kernel(0)
    try:
        assert kernels(lambda: mlp.forward_mlp_prepared(x)) == {"ffn_imma_kernel"}
        assert kernels(lambda: mlp.forward_mlp(x)) == {"ffn_imma_kernel"}
        assert kernels(lambda: ops.decode_stack([mlp], x.clone())) == {"ffn_imma_kernel"}
    finally:
        L.load().ffn_int4_set_decode_kernel(old)
        mlp.release()


@pytest.mark.parametrize("tokens", [3, 16, 64, 65, 128, 200])
def test_batched_ffn_on_one_rank(cuda, tokens):
    mlp = layer(cuda, 2560, 2176)
    mlp.dims.max_chunk = 200
    x = torch.randn((tokens, 2560), device=cuda).to(torch.bfloat16)
    assert kernels(lambda: mlp.forward_mlp_prepared(x)) == {"stream_tc_kernel"}
    assert kernels(lambda: mlp.forward_mlp(x)) == {"stream_tc_kernel"}


@pytest.mark.parametrize("rows,n,k", [(3, 12288, 5120), (3, 8, 2816), (8, 12288, 5120), (8, 2464, 2560), (7, 8, 128), (9, 264, 256),
                                      (128, 4104, 1280), (513, 520, 512)])
def test_gemm(cuda, rows, n, k):
    packed, scales = ops.quantize_int4(torch.empty((n, k), device=cuda).normal_(0.0, 0.02))
    a = torch.randn((rows, k), device=cuda).to(torch.bfloat16)
    assert kernels(lambda: ops.gemm_int4_bf16(a, packed, scales)) == {"stream_tc_kernel"}


@pytest.mark.parametrize("rows,n,k", [(3, 2048, 2560), (4, 4096, 2560), (5, 8, 128), (6, 264, 256), (8, 2456, 2560)])
def test_gemm_of_a_few_rows_and_a_small_matrix(cuda, rows, n, k):
    packed, scales = ops.quantize_int4(torch.empty((n, k), device=cuda).normal_(0.0, 0.02))
    a = torch.randn((rows, k), device=cuda).to(torch.bfloat16)
    assert kernels(lambda: ops.gemm_int4_bf16(a, packed, scales)) == {"gemm_int4_rows_kernel"}
    want = a.double() @ ops.dequantize_int4(packed, scales)[0].double().T
    # half a BF16 ulp, and sums in FP32 of a few hundred terms each: far below that ulp
    assert (ops.gemm_int4_bf16(a, packed, scales).double() - want).norm() / want.norm() <= 2.0 ** -8
