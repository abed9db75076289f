"""The GPU quantizer's rounding where the quotient is a half or next to one, at scales from the smallest to the
largest that the format holds, byte for byte against the CPU oracle; and the ways of delivering the bytes: through
scratch in 16-byte or in 2-byte pieces, and by a second pass."""
import numpy as np
import pytest
import torch

from haskell_infer_demo_b200 import lib as L
from haskell_infer_demo_b200 import ops
from oracle import ffn_oracle as o

pytestmark = pytest.mark.gpu


def same(w, cuda):
    packed, scales = ops.quantize_int4(torch.from_numpy(w).to(cuda))
    want_p, want_s = o.quantize(w)
    assert np.array_equal(packed.cpu().numpy(), want_p)
    assert np.array_equal(scales.view(torch.int16).cpu().numpy().view(np.uint16), want_s)


@pytest.mark.parametrize("exponent", [-133, -130, -126, -101, -100, -99, -20, 0, 100, 125])
def test_halves_and_their_neighbours(cuda, exponent):
    rng = np.random.default_rng(exponent + 200)
    rows = []
    for mant in range(128, 256, 5):                              # BF16 scales mant * 2^(exponent - 7)
        scale = np.float32(np.ldexp(float(mant), exponent - 7))
        q = rng.integers(-7, 7, 127).astype(np.float64) + 0.5
        x = (q * float(scale)).astype(np.float32)
        x = np.concatenate([[np.float32(7.0) * scale], x])
        for step in (0, 1, -1, 2, -2):
            y = x.copy()
            y[1:] = (y[1:].view(np.int32) + step).view(np.float32)
            if np.isfinite(y).all() and np.abs(y).max() > 0:
                rows.append(y)
    w = np.stack(rows[:len(rows) // 8 * 8]).astype(np.float32)
    if not len(w):
        pytest.skip("the format holds no such scale")
    try:
        o.quantize(w)
    except ValueError:
        with pytest.raises(Exception):
            ops.quantize_int4(torch.from_numpy(w).to(cuda))
        return
    same(w, cuda)


@pytest.mark.parametrize("n,k", [(8, 128), (24, 384), (1032, 256), (26224, 5120)])
def test_random_matrices_through_scratch_and_past_it(cuda, n, k):
    """26224 x 5120 is 67 MB of bytes, more than the scratch takes."""
    same(np.random.default_rng(n).standard_normal((n, k), dtype=np.float32) * np.float32(0.02), cuda)


@pytest.mark.parametrize("n,k", [(8, 128), (1032, 256), (26224, 5120)])
def test_outputs_off_their_alignment(cuda, n, k):
    """Outputs at a 2-byte offset receive the same bytes, and a refused matrix leaves them and their surroundings
    alone.  The third size is past what the scratch takes."""
    gen = torch.Generator(device=cuda).manual_seed(n)
    w = torch.empty((n, k), device=cuda).normal_(0.0, 0.02, generator=gen)
    want_p, want_s = ops.quantize_int4(w)
    store_p = torch.full((n * k // 2 + 18,), 0xAB, dtype=torch.uint8, device=cuda)
    store_s = torch.full((n * k // 128 + 9,), 0x1234, dtype=torch.int16, device=cuda)

    def call():
        return L.load().ffn_quantize_int4(w.data_ptr(), store_p.data_ptr() + 2, store_s.data_ptr() + 2, n, k, None)

    w[n // 2, 5] = float("inf")
    torch.cuda.synchronize()
    assert call() == -3
    assert (store_p == 0xAB).all() and (store_s == 0x1234).all()
    w.normal_(0.0, 0.02, generator=gen.manual_seed(n))
    torch.cuda.synchronize()
    assert call() == 0
    assert torch.equal(store_p[2:2 + n * k // 2].view(n, -1), want_p)
    assert torch.equal(store_s[1:1 + n * k // 128].view(n, -1), want_s.view(torch.int16))
    assert (store_p[:2] == 0xAB).all() and (store_p[2 + n * k // 2:] == 0xAB).all()
    assert (store_s[:1] == 0x1234).all() and (store_s[1 + n * k // 128:] == 0x1234).all()
