"""The sorted schedule (coherence key, three-pass radix sort, ray counter) on batches of
millions of rays, against the default schedule ray by ray and against the oracle on a
sample. The sizes lie on both sides of the line between the sort's two prefix sums
(2,048 tiles of 4,096 keys)."""
import numpy as np
import pytest

from conftest import same_bits

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

SORTED, AUTO = 4, 5


@pytest.mark.parametrize("width,n", [(8, 4_194_304), (8, 4_194_305), (4, 8_388_608), (8, 8_388_609)])
def test_sorted_schedule_matches_batch_order_and_oracle(port, width, n):
    from sort_b200 import Obvh, Qbvh, scenes
    tri = scenes.sphere_field(64, 3, seed=80)
    acc = (Qbvh if width == 4 else Obvh)()
    acc.Build(tri)
    assert acc.GetTuning()["schedule"] == AUTO
    rays = scenes.random_rays(n, seed=81)
    d = torch.from_numpy(np.ascontiguousarray(rays)).cuda()
    base = acc.GetIntersect(d)
    base_occ = acc.GetAttenuation(d)
    acc.SetTuning(schedule=SORTED)
    for _ in range(2):  # the second sort reuses the first one's scratch
        h = acc.GetIntersect(d)
        occ = acc.GetAttenuation(d)
        for a, b in ((h.prim, base.prim), (h.t, base.t), (h.u, base.u), (h.v, base.v)):
            assert torch.equal(a.view(torch.int32), b.view(torch.int32))
        assert torch.equal(occ, base_occ)
    idx = np.sort(np.random.default_rng(82).choice(n, 65_536, replace=False))
    idx[-1] = n - 1
    sample = np.ascontiguousarray(rays[:, idx])
    ref = port.build(tri, width)
    prim, t, u, v = ref.closest(sample)
    got = [x.cpu().numpy()[idx] for x in (h.prim, h.t, h.u, h.v, occ)]
    assert np.array_equal(got[0], prim) and np.array_equal(got[4], ref.any(sample))
    assert same_bits(got[1], t) and same_bits(got[2], u) and same_bits(got[3], v)
    assert 0.05 < (prim >= 0).mean() < 1.0
    acc.Release()
