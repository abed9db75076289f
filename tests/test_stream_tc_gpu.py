"""The streaming tensor-core kernel (three rows and more) at the edges of its row blocks, K pieces and token
blocks: the GEMM against FP64 sums over the dequantized matrix, the FFN against the CPU oracle."""
import numpy as np
import pytest
import torch

from gpu_util import assert_ffn_close, dev_bf16, host_f32, kernels, upload_layer
from haskell_infer_demo_b200 import lib as L
from haskell_infer_demo_b200 import ops
from oracle import ffn_oracle as o

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,k", [(8, 128), (264, 256), (4104, 1280), (37896, 512), (512, 17408), (128, 640)])
@pytest.mark.parametrize("rows", [3, 16, 17, 33, 48, 64, 65, 81, 112, 128, 129, 300, 513])
def test_gemm_against_fp64(cuda, rows, n, k):
    gen = torch.Generator(device="cuda").manual_seed(rows * 100003 + n)
    packed, scales = ops.quantize_int4(torch.randn((n, k), generator=gen, device=cuda) * 0.02)
    a = torch.randn((rows, k), generator=gen, device=cuda).to(torch.bfloat16)
    # three rows of a small matrix are the shape-generic kernel's: as sharp a check of that one, then
    small = rows == 3 and k <= 2730 and rows * n * 2 <= 65536 and rows * n * k * 2 <= 48 << 20
    assert kernels(lambda: ops.gemm_int4_bf16(a, packed, scales)) in ({"gemm_int4_rows_kernel" if small else "stream_tc_kernel"}, None)
    got = ops.gemm_int4_bf16(a, packed, scales).double()
    w = ops.dequantize_int4(packed, scales)[0].double()
    want = a.double() @ w.T
    # FP32 sums: 128 products of a group (the tensor core may truncate: 2^-23 each), the groups one after the other,
    # the pieces of a block (at most the square root of its units); the generic kernel's are no deeper.  Then
    # half a BF16 ulp: 2^-8 of a value at most; over many values its root mean square, ulp / sqrt(12), is 1.7e-3 of theirs.
    groups = k // 128
    off = (a.double().abs() @ w.abs().T) * ((128 + groups + groups ** 0.5 + 1) * 2.0 ** -23)
    assert (got - want).abs().le((want.abs() + off) * 2.0 ** -8 + off).all()
    assert want.numel() < 1000 or (got - want).norm() <= want.norm() * 2.0 ** -9
    assert torch.equal(ops.gemm_int4_bf16(a, packed, scales).double(), got)     # a fixed order of summation
    L.device_status()


@pytest.mark.parametrize("hidden,inter", [(128, 128), (384, 1152), (1024, 3072), (2560, 640)])
@pytest.mark.parametrize("tokens", [3, 24, 48, 70, 128])
def test_ffn_with_norm_against_oracle(cuda, tokens, hidden, inter):
    x, layers = o.draw_config(hidden, inter, 5 + tokens, tokens=tokens, layers=1, with_norm=True)
    layer = layers[0]
    want, _, act = o.ffn(layer, o.gemma_rmsnorm(x, layer.w_norm), intermediates=True)
    mlp = upload_layer(layer, cuda, with_norm=True)
    ws = mlp.workspace(tokens)
    xd = dev_bf16(x, cuda)
    assert kernels(lambda: mlp.forward_mlp(xd, ws=ws)) in ({"stream_tc_kernel"}, None)
    got = mlp.forward_mlp(xd, ws=ws)
    L.device_status()
    assert_ffn_close(host_f32(got), want, f"{hidden}x{inter} M={tokens}")
    left = host_f32(ws[tokens * (hidden + 2 * inter):tokens * (hidden + 3 * inter)].view(tokens, inter))
    assert o.compare(left, act)[1] <= 5e-3


def test_more_tokens_than_one_launch_takes(cuda):
    """600 tokens are a launch of 512 and one of 88: every row as its own small call gives it."""
    _, layers = o.draw_config(512, 640, 3, tokens=1, layers=1)
    mlp = upload_layer(layers[0], cuda)
    mlp.dims.max_chunk = 600
    x = torch.randn((600, 512), device=cuda).to(torch.bfloat16)
    got = mlp.forward_mlp_prepared(x)
    for m in range(0, 600, 100):
        want = mlp.forward_mlp_prepared(x[m:m + 100].contiguous())
        # the split of K over CTAs differs with the number of tokens: FP32 order, then BF16 roundings of act and y
        err = (got[m:m + 100].float() - want.float()).norm() / want.float().norm()
        assert err <= 2.0 ** -8
    L.device_status()


def test_scales_off_their_alignment(cuda):
    """Scales at a 2-byte offset are read one by one, with the same result."""
    packed, scales = ops.quantize_int4(torch.randn((1048, 2048), device=cuda) * 0.02)
    store = torch.empty(scales.numel() + 1, dtype=torch.bfloat16, device=cuda)
    off = store[1:].view(scales.shape)
    off.copy_(scales)
    for rows in (9, 100):
        a = torch.randn((rows, 2048), device=cuda).to(torch.bfloat16)
        assert torch.equal(ops.gemm_int4_bf16(a, packed, off), ops.gemm_int4_bf16(a, packed, scales))
    L.device_status()


def test_a_row_with_nan_stays_alone(cuda):
    packed, scales = ops.quantize_int4(torch.randn((520, 640), device=cuda) * 0.02)
    a = torch.randn((21, 640), device=cuda).to(torch.bfloat16)
    want = ops.gemm_int4_bf16(a, packed, scales)
    a[9, 333] = float("nan")
    got = ops.gemm_int4_bf16(a, packed, scales)
    assert got[9].isnan().all()
    keep = [m for m in range(21) if m != 9]
    assert torch.equal(got[keep], want[keep])
    assert np.isfinite(host_f32(got[keep])).all()
