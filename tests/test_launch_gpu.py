"""A decode call whose CTAs have to wait for SMs: a launch is only once, at first, made for the whole GPU at a time, later ones
come to the SMs as they become free.  With another stream's kernels on all SMs the results are the same, and no wait runs out."""
import pytest
import torch

from haskell_infer_demo_b200 import lib as L
from haskell_infer_demo_b200 import ops
from test_stack_launch_gpu import layers_of, same

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tokens", [1, 2])
@pytest.mark.parametrize("hidden,inter", [(256, 1024), (5120, 2176), (2560, 9728)])
def test_next_to_kernels_on_every_sm(cuda, tokens, hidden, inter):
    mlps, draw = layers_of(cuda, hidden, inter, 3)
    x, h0 = draw(tokens), draw(tokens)

    def call():
        h = h0.clone()
        ops.decode_stack(mlps, h)
        return [m.forward_mlp_prepared(x).clone() for m in mlps], h

    want, want_h = call()
    torch.cuda.synchronize()
    a = torch.randn((8192, 8192), device=cuda, dtype=torch.bfloat16)
    other = torch.cuda.Stream()
    other.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(other):
        for _ in range(40):
            a @ a
    for _ in range(20):
        ys, h = call()
        assert same(h, want_h) and all(same(y, w) for y, w in zip(ys, want))
    torch.cuda.synchronize()
    L.device_status()


def test_two_launches_in_a_graph(cuda):
    mlps, draw = layers_of(cuda, 1024, 3072, 2)
    x = draw(1)
    ws, out = mlps[0].workspace(1), [torch.empty_like(x) for _ in mlps]
    want = [m.forward_mlp_prepared(x).clone() for m in mlps]
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        for _ in range(3):
            for m, o in zip(mlps, out):
                m.forward_mlp_prepared(x, ws, o)
    for _ in range(5):
        graph.replay()
    torch.cuda.synchronize()
    L.device_status()
    assert all(same(o, w) for o, w in zip(out, want))
