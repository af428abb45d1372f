"""The walk of small launches (group_walk.cuh, eight lanes per ray) at the edges of
its launch shapes: a ray per warp, a share of each warp's groups, a ray per group,
and one ray more, which the walk of large launches takes; leaves shorter and longer
than eight triangles, rays with tmin <= -1. FP32 nodes match the oracle bit for bit;
every prefix of a batch matches the whole batch bit for bit."""
import numpy as np
import pytest

from conftest import same_bits

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("nodes", ["fp32", "q8"])
@pytest.mark.parametrize("max_leaf,stack", [(8, 16), (33, 100)])
def test_small_launches(port, nodes, max_leaf, stack):
    from sort_b200 import Obvh, _lib, scenes
    from test_gpu_walk import stacked
    warps = torch.cuda.get_device_properties(0).multi_processor_count * 32
    limit = warps * 4
    tri = np.concatenate([stacked(stack, 60 + stack), scenes.sphere_field(16, 3, seed=61)])
    fmt = _lib.SG_NODES_QUANT8 if nodes == "q8" else _lib.SG_NODES_FP32
    acc = Obvh(max_pri_in_leaf=max_leaf, node_format=fmt)
    acc.Build(tri)
    rays = scenes.random_rays(limit + 1, seed=62)
    rays[6, ::3] = -1.0
    rays[6, 1::7] = -25.0
    rays[7, ::5] = 0.75
    d = torch.from_numpy(np.ascontiguousarray(rays)).cuda()

    def run(n):
        part = d[:, :n].contiguous()
        h, occ = acc.GetIntersect(part), acc.GetAttenuation(part)
        torch.cuda.synchronize()
        return [x.cpu().numpy() for x in (h.prim, h.t, h.u, h.v, occ)]

    whole = run(limit + 1)
    if nodes == "fp32":
        ref = port.build(tri, 8, 16, max_leaf)
        prim, t, u, v = ref.closest(rays)
        assert np.array_equal(whole[0], prim) and np.array_equal(whole[4], ref.any(rays))
        assert all(same_bits(a, b) for a, b in zip(whole[1:4], (t, u, v)))
    for n in (1, 2, 33, warps - 1, warps, warps + 1, 2 * warps - 1, limit - 1, limit):
        part = run(n)
        assert np.array_equal(part[0], whole[0][:n]) and np.array_equal(part[4], whole[4][:n])
        assert all(same_bits(a, b[:n]) for a, b in zip(part[1:4], whole[1:4]))
