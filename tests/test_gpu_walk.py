"""The warp-cooperative traversal (warp_walk.cuh) where its shape can go wrong:
leaves shorter and longer than the eight lanes that test one, batch sizes around
the line between equal shares and a ray counter, rays with tmin <= -1 (SORT's
rule for three and more hit children), captured and concurrent launches. Hits,
distances and barycentrics are the oracle's bit for bit."""
import numpy as np
import pytest

from conftest import same_bits

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def accel(width, **kw):
    from sort_b200 import Obvh, Qbvh
    return (Qbvh if width == 4 else Obvh)(**kw)


def check(acc, ref, rays):
    d = torch.from_numpy(np.ascontiguousarray(rays)).cuda()
    h = acc.GetIntersect(d)
    occ = acc.GetAttenuation(d)
    torch.cuda.synchronize()
    prim, t, u, v = ref.closest(rays)
    assert np.array_equal(h.prim.cpu().numpy(), prim)
    assert same_bits(h.t.cpu().numpy(), t) and same_bits(h.u.cpu().numpy(), u) and same_bits(h.v.cpu().numpy(), v)
    assert np.array_equal(occ.cpu().numpy(), ref.any(rays))


def stacked(n, seed):
    """n triangles with one box (no split separates them; every third is a copy,
    hit at the same distance), then a sphere field."""
    from sort_b200 import scenes
    z = np.linspace(-1.0, 1.0, n)
    z[::3] = z[0]
    tri = np.zeros((n, 3, 3))
    tri[:, 0] = (-2.0, -2.0, 1.0)
    tri[:, 1] = (2.0, -2.0, -1.0)
    tri[:, 2, 1] = 4.0
    tri[:, 2, 2] = z
    return np.concatenate([tri.reshape(-1, 9).astype(np.float32), scenes.sphere_field(4, 2, seed=seed)])


@pytest.mark.parametrize("width", [4, 8])
@pytest.mark.parametrize("max_leaf,stack", [(1, 1), (7, 7), (8, 16), (9, 17), (33, 100)])
def test_leaf_sizes(port, width, max_leaf, stack):
    from sort_b200 import scenes
    tri = stacked(stack, 40 + stack)
    acc = accel(width, max_pri_in_leaf=max_leaf)
    acc.Build(tri)
    rays = np.concatenate([scenes.camera_rays(64, 64, seed=41), scenes.random_rays(4096, seed=42)], axis=1)
    check(acc, port.build(tri, width, 16, max_leaf), rays)


@pytest.mark.parametrize("width", [4, 8])
def test_batch_sizes_and_negative_tmin(port, width):
    from sort_b200 import scenes
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    line = sms * (7 if width == 8 else 8) * 4 * 32  # rays that fill every resident warp once
    tri = scenes.sphere_field(32, 3, seed=43)
    acc = accel(width)
    acc.Build(tri)
    ref = port.build(tri, width)
    rays = scenes.random_rays(line + 65, seed=44)
    rays[6, ::3] = -1.0   # at and below -1, SORT drops children at distances <= -1 when three or more are hit
    rays[6, 1::7] = -25.0
    for n in (1, 31, 33, sms * 28 + 1, line - 1, line, line + 1, line + 65):
        check(acc, ref, rays[:, :n])


def test_captured_and_concurrent_launches(port):
    """A captured launch takes no scratch, so its graph may be replayed beside
    other launches; large launches on several streams share nothing."""
    from sort_b200 import scenes
    tri = scenes.sphere_field(32, 3, seed=45)
    acc = accel(8)
    acc.Build(tri)
    rays = scenes.random_rays(300_001, seed=46)
    want = port.build(tri, 8).closest(rays)
    d = torch.from_numpy(rays).cuda()
    for _ in range(2):  # any-hit and closest-hit kernels loaded before the capture
        acc.GetAttenuation(d)
        acc.GetIntersect(d)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        captured = acc.GetIntersect(d)
    streams = [torch.cuda.Stream() for _ in range(3)]
    results = []
    for rep in range(3):
        graph.replay()
        for s in streams:
            s.wait_stream(torch.cuda.current_stream()) if rep == 0 else None
            with torch.cuda.stream(s):
                results.append(acc.GetIntersect(d))
    torch.cuda.synchronize()
    for h in [captured] + results:
        assert np.array_equal(h.prim.cpu().numpy(), want[0]) and same_bits(h.t.cpu().numpy(), want[1])


@pytest.mark.parametrize("sizes", [(1,), (33, 0, 5), (4_000, 7), (140_001, 1, 3)])
def test_batch_groups_smaller_and_larger_than_the_grid(sizes):
    """A group of fewer rays than the grid has lanes is claimed in equal shares,
    a larger one from its counter: each batch's answers are its own launch's."""
    from sort_b200 import Batch, Batcher, scenes
    accs = []
    for width, seed in ((8, 47), (4, 48)):
        accs.append(accel(width))
        accs[-1].Build(scenes.sphere_field(16, 2, seed=seed))
    pool = torch.from_numpy(scenes.random_rays(150_000, seed=49)).cuda()
    batches = [Batch(a, pool[:, k:k + n], any=q) for a in accs for q in (False, True) for k, n in enumerate(sizes)]
    batcher = Batcher(max_batches=32)
    for _ in range(2):
        batcher.run(batches)
        done = batcher.wait()
        assert (done[: len(batches)] >= 0).all()
        for b in batches:
            if b.rays.shape[1] == 0:
                continue
            if b.any:
                assert torch.equal(b.occluded, b.accel.GetAttenuation(b.rays))
            else:
                h = b.accel.GetIntersect(b.rays)
                assert torch.equal(b.hits.prim, h.prim) and torch.equal(b.hits.t.view(torch.int32), h.t.view(torch.int32))
    batcher.Release()
