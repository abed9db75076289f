"""The GPU quantizer's rounding where the quotient is a half or next to one, at scales from the smallest to the
largest that the format holds, and both ways of delivering the bytes: byte for byte against the CPU oracle."""
import numpy as np
import pytest
import torch

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
