"""Small nodes of the GPU builder (split by one warp each) around the line where
they take over from the rounds: SORT's tree, primitive for primitive, and the
host build's node numbering."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

SMALL = 1024  # the builder's kSmall


def soup(n, seed, kind):
    rng = np.random.default_rng(seed)
    c = rng.uniform(-10.0, 10.0, (n, 1, 3))
    if kind == "clusters":  # ranges that bins cannot separate, next to ones they can
        c = rng.integers(-3, 4, (n, 1, 3)).astype(np.float64)
    elif kind == "plane":
        c[:, :, 1] = 0.25
    elif kind == "line":
        c[:, :, :2] = 0.0
        c[:, 0, 2] = np.exp(rng.uniform(-12.0, 3.0, n))
    tri = c + rng.uniform(-0.3, 0.3, (n, 3, 3)) * (0.0 if kind == "clusters" else 1.0)
    if kind == "clusters":
        tri = tri + np.array([[[-0.5, 0.0, 0.0], [0.5, 0.0, 0.25], [0.0, 0.5, -0.25]]])
    return np.ascontiguousarray(tri.reshape(n, 9).astype(np.float32))


@pytest.mark.parametrize("width", [4, 8])
@pytest.mark.parametrize("kind", ["uniform", "clusters", "plane", "line"])
@pytest.mark.parametrize("n", [2, 9, 33, SMALL - 1, SMALL, SMALL + 1, 3 * SMALL + 5, 40_000])
def test_small_nodes_build_sorts_tree(width, kind, n):
    from sort_b200 import Obvh, Qbvh, _lib, build_topology_host, scenes
    cls = Qbvh if width == 4 else Obvh
    tri = soup(n, 60 + n % 7, kind)
    rays = torch.from_numpy(scenes.random_rays(2048, seed=61)).cuda()
    for max_leaf, max_depth in ((8, 16), (1, 16), (3, 5)):
        topo, depth = build_topology_host(tri, width, max_depth, max_leaf)
        got = []
        for builder in (_lib.SG_BUILDER_GPU, _lib.SG_BUILDER_HOST):
            acc = cls(max_depth, max_leaf, builder=builder)
            acc.Build(tri)
            assert np.array_equal(acc.topology(), topo) and acc.info()["depth"] == depth
            h = acc.GetIntersect(rays)
            got.append((acc.info()["interior_nodes"], acc.info()["leaves"], h))
            acc.Release()
        assert got[0][:2] == got[1][:2]
        for a, b in zip((got[0][2].prim, got[0][2].t), (got[1][2].prim, got[1][2].t)):
            assert torch.equal(a, b)
