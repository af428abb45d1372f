"""Leaves of the Morton-order trees (LBVH, PLOC), filled after the collapse: every
primitive lies in exactly one leaf, no leaf is larger than max_leaf, on both sides
of the size up to which a leaf is walked with a stack, and the trees find the hits
SORT's tree finds (up to near-ties, which the sphere fields of this test lack on
all but a handful of rays)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def leaves(topo):
    out, k = [], 0
    stack = 1
    while stack:
        stack -= 1
        children = int(topo[k])
        k += 1
        if children:
            stack += children
        else:
            n = int(topo[k])
            out.append(topo[k + 1:k + 1 + n])
            k += 1 + n
    assert k == len(topo)
    return out


@pytest.mark.parametrize("width", [4, 8])
@pytest.mark.parametrize("builder", ["SG_BUILDER_LBVH", "SG_BUILDER_PLOC"])
@pytest.mark.parametrize("max_leaf", [1, 2, 8, 15, 16, 17, 64])
def test_every_primitive_in_one_leaf(width, builder, max_leaf):
    from sort_b200 import Obvh, Qbvh, _lib, scenes
    cls = Qbvh if width == 4 else Obvh
    tri = scenes.sphere_field(12, 3, seed=70)
    rays = torch.from_numpy(scenes.random_rays(20_000, seed=71)).cuda()
    ref = cls()
    ref.Build(tri)
    want = ref.GetIntersect(rays)
    acc = cls(max_pri_in_leaf=max_leaf, builder=getattr(_lib, builder))
    acc.Build(tri)
    parts = leaves(acc.topology())
    assert max(len(p) for p in parts) <= max_leaf and len(parts) == acc.info()["leaves"]
    assert np.array_equal(np.sort(np.concatenate(parts)), np.arange(len(tri)))
    got = acc.GetIntersect(rays)
    same = (got.prim == want.prim) & (got.t == want.t)
    assert int((~same).sum()) <= 20
