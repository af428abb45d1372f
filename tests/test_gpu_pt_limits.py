"""Frames and pools at the size limits: places in a wave's shadow queue (two rays per
path, eight planes) are ints, so a wave holds at most 2^27 paths and a larger frame
takes several waves per sample; a server's pool holds no more slots. A request's rows
may be longer than a server's pool has slots."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.fixture(scope="module")
def tracer():
    from sort_b200 import scenes
    from sort_b200.pathtracer import PathTracer
    _, _, mats, light, tri, mat = scenes.pt_scene(12, 2, seed=3)
    pt = PathTracer(tri, mat, mats, light)
    yield pt
    pt.Release()
    torch.cuda.empty_cache()


def test_frame_beyond_one_wave_is_its_bands(tracer):
    """153.8M pixels: 14 times that, the last plane of the shadow queue, is beyond 2^31."""
    from sort_b200 import scenes
    side = 12_400
    assert 7 * 2 * side * side > 2**31
    whole = tracer.Render(scenes.CAMERA, side, side, 1, 2, seed=5)
    rays = np.array(tracer.RayCounts())
    total = np.zeros(2, np.int64)
    for a, b in ((0, side // 2), (side // 2, side)):
        band = tracer.Render(scenes.CAMERA, side, side, 1, 2, seed=5, rows=(a, b))
        assert torch.equal(band, whole[a:b])
        total += np.array(tracer.RayCounts())
        del band
    assert np.array_equal(rays, total) and float(whole.mean()) > 0


def test_largest_pool_renders_the_same_image(tracer):
    from sort_b200 import scenes
    from sort_b200.server import RenderServer
    want = tracer.Render(scenes.CAMERA, 64, 36, 2, 5, seed=6).cpu().numpy()
    srv = RenderServer(path_slots=1 << 28, pixel_budget=1 << 16, solo_pixels=-1)
    try:
        sid = srv.add_scene(tracer)
        img, res = srv.wait(srv.submit(sid, scenes.CAMERA, 64, 36, 2, 5, seed=6))
        assert res["status"] == 0 and np.array_equal(img.view(np.int32), want.view(np.int32))
    finally:
        srv.close()


@pytest.mark.parametrize("spp", [1, 3])
def test_rows_longer_than_the_pool(tracer, spp):
    from sort_b200 import scenes
    from sort_b200.server import RenderServer
    want = tracer.Render(scenes.CAMERA, 201, 3, spp, 4, seed=7).cpu().numpy()
    srv = RenderServer(path_slots=64, pixel_budget=1 << 12)
    try:
        sid = srv.add_scene(tracer)
        for _ in range(2):
            img, res = srv.wait(srv.submit(sid, scenes.CAMERA, 201, 3, spp, 4, seed=7))
            assert res["status"] == 0 and np.array_equal(img.view(np.int32), want.view(np.int32))
    finally:
        srv.close()
