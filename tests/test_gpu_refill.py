"""Refilled lanes: a batch larger than the GPU's resident lanes, so that warps take
rays again and again, under every refill threshold that matters, without a counter
(captured launches go by spans), and with NaN and infinite rays among the ones taken.
FP32 nodes give the oracle's bits; 8-bit nodes the bits of their own default launch."""
import numpy as np
import pytest

from conftest import same_bits

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

N = 300_001  # above 148 SMs x 8 blocks x 128 lanes, with a remainder


def build(width, q8, tri):
    from sort_b200 import Obvh, Qbvh, _lib
    acc = (Qbvh if width == 4 else Obvh)(node_format=_lib.SG_NODES_QUANT8 if q8 else _lib.SG_NODES_FP32)
    acc.Build(tri)
    return acc


def answers(acc, d):
    h, occ = acc.GetIntersect(d), acc.GetAttenuation(d)
    torch.cuda.synchronize()
    return [x.cpu().numpy() for x in (h.prim, h.t, h.u, h.v, occ)]


def same(a, b):
    return all(same_bits(x, y) if x.dtype == np.float32 else np.array_equal(x, y) for x, y in zip(a, b))


def more_rays_than_lanes():
    p = torch.cuda.get_device_properties(0)
    assert N > p.multi_processor_count * 8 * 128


@pytest.mark.parametrize("q8", [False, True])
@pytest.mark.parametrize("width", [4, 8])
def test_refill_thresholds_and_spans(port, width, q8):
    from sort_b200 import scenes
    more_rays_than_lanes()
    tri = scenes.sphere_field(32, 3, seed=85)
    rays = scenes.random_rays(N, seed=86)
    d = torch.from_numpy(np.ascontiguousarray(rays)).cuda()
    acc = build(width, q8, tri)
    want = answers(acc, d)
    if not q8:
        ref = port.build(tri, width)
        assert same(want, [*ref.closest(rays), ref.any(rays)])
    for refill in (1, 8, 31, 32):
        acc.SetTuning(1, refill)  # SG_SCHEDULE_PERSISTENT
        assert same(answers(acc, d), want), refill
    acc.SetTuning(5, 8)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):  # no counter: spans of rays per warp
        h, occ = acc.GetIntersect(d), acc.GetAttenuation(d)
    for _ in range(2):
        graph.replay()
    torch.cuda.synchronize()
    assert same([x.cpu().numpy() for x in (h.prim, h.t, h.u, h.v, occ)], want)
    del graph
    acc.Release()
