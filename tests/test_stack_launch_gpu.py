"""A stack of one or two tokens in one launch: the same bits as its layers called one after the other, over the edges of
its plans (one and two column chunks a thread in either phase, hidden sizes on both sides of the intermediate one,
ragged tiles, ragged shares of rows), more layers than a launch holds, replays of a captured graph, and a call that it
leaves to the single-layer kernel."""
import pytest
import torch

from haskell_infer_demo_b200 import lib as L
from haskell_infer_demo_b200 import ops
from test_routes_gpu import kernels

pytestmark = pytest.mark.gpu


def layers_of(cuda, hidden, inter, count, seed=3):
    gen = torch.Generator(device=cuda).manual_seed(seed)

    def q(n, k):
        return ops.quantize_int4(torch.empty((n, k), device=cuda).normal_(0.0, 0.02, generator=gen))

    def norm():
        return torch.randn(hidden, generator=gen, device=cuda).mul_(0.1).to(torch.bfloat16)

    return [ops.DenseMlp(*q(2 * inter, hidden), *q(hidden, inter), post_norm_w=norm()) for _ in range(count)], \
        lambda tokens: torch.randn((tokens, hidden), generator=gen, device=cuda).to(torch.bfloat16)


def one_by_one(mlps, h0):
    h, y = h0.clone(), torch.empty_like(h0)
    for m in mlps:
        ops.decode_stack([m], h, layer_out=y)
    L.device_status()
    return h, y


def same(a, b):
    return torch.equal(a.view(torch.int16), b.view(torch.int16))


@pytest.mark.parametrize("tokens", [1, 2])
@pytest.mark.parametrize("hidden,inter,count", [(256, 256, 2), (256, 1024, 5), (1024, 3072, 3), (2560, 9728, 3), (8192, 512, 2),
                                                (5120, 2176, 3), (512, 17408, 2), (1024, 384, 65), (4096, 14336, 2)])
def test_equals_its_layers(cuda, tokens, hidden, inter, count):
    mlps, draw = layers_of(cuda, hidden, inter, count)
    h0 = draw(tokens)
    want_h, want_y = one_by_one(mlps, h0)
    for _ in range(3):
        h, y = h0.clone(), torch.empty_like(h0)
        ops.decode_stack(mlps, h, layer_out=y)
        L.device_status()
        assert same(h, want_h) and same(y, want_y)
    h = h0.clone()
    assert kernels(lambda: ops.decode_stack(mlps, h)) == {"ffn_stack_kernel"}


def test_a_captured_stack_replays(cuda):
    mlps, draw = layers_of(cuda, 1024, 3072, 4)
    h0 = draw(1)
    want, _ = one_by_one(mlps, h0)
    h, ws, y = h0.clone(), mlps[0].workspace(1), torch.empty_like(h0)
    ops.decode_stack(mlps, h, ws=ws, layer_out=y)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        ops.decode_stack(mlps, h, ws=ws, layer_out=y)
    for _ in range(3):
        h.copy_(h0)
        graph.replay()
        torch.cuda.synchronize()
        L.device_status()
        assert same(h, want)


def test_calls_between_stacks(cuda):
    """The arrivals that a stack leaves behind are what the single-layer kernel counts from, and the other way round."""
    mlps, draw = layers_of(cuda, 1024, 3072, 3)
    h0 = draw(1)
    want, _ = one_by_one(mlps, h0)
    x = draw(2)
    y = mlps[0].forward_mlp_prepared(x).clone()
    for _ in range(5):
        h = h0.clone()
        ops.decode_stack(mlps, h)
        assert same(mlps[0].forward_mlp_prepared(x), y)
        assert same(h, want)
    L.device_status()


def test_fewer_rows_than_blocks_go_layer_by_layer(cuda):
    mlps, draw = layers_of(cuda, 128, 1024, 2)
    h0 = draw(1)
    want, _ = one_by_one(mlps, h0)
    h = h0.clone()
    ops.decode_stack(mlps, h)
    L.device_status()
    assert same(h, want)
