"""NaN and infinite rays on the walks that a few thousand rays do not leave (eight lanes
per ray over width-8 trees, one ray per warp over width-4 ones) and on refilled lanes.
Such rays can reach empty child slots. FP32 nodes give the oracle's answers; 8-bit
nodes the same ones in a small and a large launch."""
import numpy as np
import pytest

from conftest import same_bits
from test_gpu_refill import N, answers, build, more_rays_than_lanes, same

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

SMALL = 4_099


def rays_with_non_finite(n, seed):
    """Every third ray has one to four bad components, each of the eight alone among
    the first of them."""
    from sort_b200 import scenes
    rng = np.random.default_rng(seed)
    rays = scenes.random_rays(n, seed=seed).copy()
    vals = np.array([np.nan, np.inf, -np.inf], np.float32)
    for k, j in enumerate(range(0, n, 3)):
        if k < 24 * 8:
            rays[k % 8, j] = vals[k // 8 % 3]
        else:
            comps = rng.choice(8, size=rng.integers(1, 5), replace=False)
            rays[comps, j] = rng.choice(vals, size=comps.size)
    return rays


@pytest.mark.parametrize("q8", [False, True])
@pytest.mark.parametrize("width", [4, 8])
def test_non_finite_rays(port, width, q8):
    from sort_b200 import scenes
    more_rays_than_lanes()
    tri = scenes.sphere_field(32, 3, seed=87)
    rays = rays_with_non_finite(N, 88)
    d = torch.from_numpy(np.ascontiguousarray(rays)).cuda()
    acc = build(width, q8, tri)
    large = answers(acc, d)
    if not q8:
        ref = port.build(tri, width)
        prim, t, _, _ = ref.closest(rays)
        assert np.array_equal(large[0], prim) and same_bits(large[1], t)
        assert np.array_equal(large[4], ref.any(rays))
        assert 0 < (prim[::3] >= 0).sum() and (prim >= 0).mean() < 1.0
    for first in (0, SMALL, N - SMALL):
        part = answers(acc, d[:, first:first + SMALL].contiguous())
        assert same(part, [x[first:first + SMALL] for x in large])
    acc.SetTuning(1, 1)  # a refill at every idle lane
    assert same(answers(acc, d), large)
    acc.Release()
