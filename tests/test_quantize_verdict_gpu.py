"""The quantizer's verdict, whose words serve one call after the other: refusals and good matrices in turn, from one thread and
from more threads, each with a stream of its own, than there are words; matrices past the scratch's size among them."""
import threading

import pytest
import torch

from haskell_infer_demo_b200 import lib as L

pytestmark = pytest.mark.gpu


def call(w, packed, scales, stream):
    return L.load().ffn_quantize_int4(w.data_ptr(), packed.data_ptr(), scales.data_ptr(), w.shape[0], w.shape[1], stream.cuda_stream)


@pytest.mark.parametrize("threads", [1, 3, 12])
@pytest.mark.parametrize("n,k", [(8, 128), (1032, 256), (26224, 5120)])
def test_refused_and_taken_in_turn(cuda, threads, n, k):
    gen = torch.Generator(device=cuda).manual_seed(n)
    good = torch.empty((n, k), device=cuda).normal_(0.0, 0.02, generator=gen)
    not_finite, too_small = good.clone(), good.clone()
    not_finite[n - 1, k - 1] = float("nan")
    too_small[n // 2, :128] = 1e-40
    blank = lambda: (torch.full((n, k // 2), 0xAB, dtype=torch.uint8, device=cuda), torch.full((n, k // 128), 0x1234, dtype=torch.int16, device=cuda))
    want = blank()
    assert call(good, *want, torch.cuda.current_stream()) == 0
    torch.cuda.synchronize()
    wrong = []

    def work():
        stream = torch.cuda.Stream()
        with torch.cuda.stream(stream):
            out, kept = blank(), blank()
            stream.synchronize()
            for _ in range(4 if n > 20000 else 20):
                for w, status in ((good, 0), (not_finite, -3), (too_small, -3), (good, 0)):
                    got = call(w, *(out if status == 0 else kept), stream)
                    if got != status:
                        wrong.append((got, status))
            if not (torch.equal(out[0], want[0]) and torch.equal(out[1], want[1]) and (kept[0] == 0xAB).all() and (kept[1] == 0x1234).all()):
                wrong.append("bytes")

    if threads == 1:
        work()
    else:
        pool = [threading.Thread(target=work) for _ in range(threads)]
        for t in pool:
            t.start()
        for t in pool:
            t.join()
    assert not wrong
