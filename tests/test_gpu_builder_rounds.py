"""The GPU builder's bound on its rounds: ranges that no cut separates are set aside,
which takes a round each beside the splits, in every node of a deep chain."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def chain(clusters, each, step):
    """Clusters of `each` triangles with one centroid at x = step^k, sized in proportion:
    every split takes the farthest cluster off the rest, and no cut splits a cluster."""
    x = np.float64(step) ** np.arange(clusters) * 1e-12
    tri = np.array([[-0.01, -0.01, 0.0], [0.01, -0.01, 0.0], [0.0, 0.02, 0.0]])[None] * x[:, None, None]
    tri[:, :, 0] += x[:, None]
    return np.ascontiguousarray(np.repeat(tri, each, axis=0).reshape(-1, 9).astype(np.float32))


@pytest.mark.parametrize("width,max_depth", [(4, 10), (4, 16), (8, 6), (8, 16)])
def test_chain_of_clusters_builds_sorts_tree(width, max_depth):
    from sort_b200 import Obvh, Qbvh, _lib, build_topology_host
    tri = chain(30, 400, 8.0)
    topo, depth = build_topology_host(tri, width, max_depth, 8)
    acc = (Qbvh if width == 4 else Obvh)(max_depth, 8, builder=_lib.SG_BUILDER_GPU)
    acc.Build(tri)
    assert np.array_equal(acc.topology(), topo) and acc.info()["depth"] == depth
    acc.Release()
