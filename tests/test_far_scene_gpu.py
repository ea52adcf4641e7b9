"""Ray queries into a small scene far from the world's origin: over the 4-wide BVH (default) and over the
BVH2 (option bvh4 = 0) every ray finds the same, bit for bit, whatever the length of its direction."""
import numpy as np
import pytest

from open_rendering_framework_b200 import _native as nat
from open_rendering_framework_b200 import scene as sc
from open_rendering_framework_b200 import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("half", [1e-3, 1e-6])
def test_small_scene_far_from_the_origin(half):
    import torch

    base = scenes.single_scene(8, 8, 1, 1)
    p = np.array([(0, -1, -1), (0, 1, -1), (0, 1, 1), (0, -1, 1)], np.float64) * half + (1000.0, 0.0, 0.0)
    wall = sc.Mesh(p.astype(np.float32), np.array([(0, 1, 2), (0, 2, 3)], np.int32), base.meshes[0].material)
    R = sc.Renderer(sc.SceneData(base.integrator, base.camera, base.background, [wall], [sc.PointLight((0.0, 0.0, 0.0), (1.0, 1.0, 1.0))]))
    rng = np.random.default_rng(4)
    n = 20_000
    o, d = np.zeros((n, 4), np.float32), np.zeros((n, 4), np.float32)
    o[:, 1:3] = rng.uniform(-half, half, (n, 2))
    d[:, 0] = 10.0 ** rng.uniform(-12.0, 0.0, n)
    d[:, 3] = 1e27
    ot, dt = torch.from_numpy(o).cuda(), torch.from_numpy(d).cuda()
    got = []
    for wide in (1, 0):
        R.set_option("bvh4", wide)
        prim, hit = (torch.full((n,), 7, dtype=torch.int32, device="cuda") for _ in range(2))
        t, b = torch.zeros(n, device="cuda"), torch.zeros((n, 2), device="cuda")
        torch.cuda.synchronize()
        nat.call("pt_trace_closest", R.ctx, ot.data_ptr(), dt.data_ptr(), n, prim.data_ptr(), t.data_ptr(), b.data_ptr())
        nat.call("pt_trace_any", R.ctx, ot.data_ptr(), dt.data_ptr(), n, hit.data_ptr())
        R.sync()
        got.append([prim.cpu().numpy(), hit.cpu().numpy(), t.cpu().numpy().view(np.uint32), b.cpu().numpy().view(np.uint32)])
    R.close()
    for a, b in zip(*got):
        assert np.array_equal(a, b)
    assert (got[1][0] >= 0).mean() > 0.99
