"""Waves of several samples: a frame rendered in waves of 4 + 1 samples, in one
wave of 5, and in bands whose waves hold other numbers of samples is the same
image, bit for bit, with the same ray counts."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("width,height,spp", [(600, 400, 5), (33, 7, 9), (1, 1, 3)])
def test_waves_of_several_samples_give_the_same_image(width, height, spp):
    from sort_b200 import scenes
    from sort_b200.pathtracer import PathTracer
    _, _, mats, light, tri, mat = scenes.pt_scene(12, 2, seed=3)
    pt = PathTracer(tri, mat, mats, light)
    whole = pt.Render(scenes.CAMERA, width, height, spp, 5, seed=11)
    rays = np.array(pt.RayCounts())
    cuts = sorted({0, 1, height // 3, height - 1, height} & set(range(height + 1)))
    bands, total = [], np.zeros(2, np.int64)
    for a, b in zip(cuts[:-1], cuts[1:]):
        bands.append(pt.Render(scenes.CAMERA, width, height, spp, 5, seed=11, rows=(a, b)))
        total += np.array(pt.RayCounts())
    assert torch.equal(torch.cat(bands).view(torch.int32), whole.view(torch.int32))
    assert np.array_equal(rays, total)
    one = pt.Render(scenes.CAMERA, width, height, 1, 5, seed=11)
    assert width * height < 100 or not torch.equal(one, whole)  # samples differ
    pt.Release()
