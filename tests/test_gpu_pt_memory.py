"""A render leaves the process most of a nearly full GPU's memory: samples share waves
only in a sixteenth of what is free, with the same image."""
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def test_small_render_on_a_nearly_full_gpu():
    from sort_b200 import scenes
    from sort_b200.pathtracer import PathTracer
    _, _, mats, light, tri, mat = scenes.pt_scene(12, 2, seed=3)
    roomy, tight = PathTracer(tri, mat, mats, light), PathTracer(tri, mat, mats, light)
    want = roomy.Render(scenes.CAMERA, 64, 36, 512, 5, seed=4)  # 455 samples a wave
    got = torch.empty_like(want)
    torch.cuda.synchronize()
    left = 2 << 30
    filler = torch.empty(torch.cuda.mem_get_info()[0] - left, dtype=torch.uint8, device="cuda")
    try:
        before = torch.cuda.mem_get_info()[0]
        assert before < 3 << 30
        for _ in range(2):
            tight.Render(scenes.CAMERA, 64, 36, 512, 5, seed=4, out=got)
            assert torch.equal(got.view(torch.int32), want.view(torch.int32))
        # What the scene holds: the driver's own memory (kernels' stacks) comes and goes beside it.
        torch.cuda.synchronize()
        held = torch.cuda.mem_get_info()[0]
        tight.Release()
        held = torch.cuda.mem_get_info()[0] - held
        assert held <= before // 16 + (16 << 20)
    finally:
        del filler
        torch.cuda.empty_cache()
        tight.Release()
        roomy.Release()
