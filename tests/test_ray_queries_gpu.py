"""Ray queries of every kind over the 4-wide BVH and over the BVH2."""
import numpy as np
import pytest

from open_rendering_framework_b200 import _native as nat
from open_rendering_framework_b200 import scene as sc
from open_rendering_framework_b200 import scenes

pytestmark = pytest.mark.gpu


def test_ray_queries_over_the_wide_bvh_match_the_bvh2_for_every_kind_of_ray():
    """pt_trace_closest / pt_trace_any over the 4-wide BVH against the BVH2 (option bvh4 = 0), bit for bit: ray
    counts around a warp's run, directions far from unit length, zero and tiny components, negative and
    infinite bounds, empty intervals, origins far away and values that are not finite."""
    import torch

    R = sc.Renderer(scenes.single_scene(8, 8, 4, 3))
    rng = np.random.default_rng(2)
    for n in (1, 31, 33, 128, 5000, 200_003):
        o = rng.uniform(-0.95, 0.95, (n, 3)).astype(np.float32)
        d = rng.normal(size=(n, 3))
        d /= np.linalg.norm(d, axis=1, keepdims=True)
        kind = np.arange(n) % 16
        d[kind == 1, 0] = 0.0
        d[kind == 2, 1:] = 0.0
        d[kind == 3] *= 1e-12
        d[kind == 4] *= 1e15
        d[kind == 5] *= 1e-30
        d[kind == 6, 2] = 1e-25
        o[kind == 7] *= 1e6
        d[kind == 8] = 0.0
        d[kind == 9, 1] = np.nan
        o[kind == 10, 0] = np.inf
        tmin, tmax = np.full(n, 1e-4, np.float32), np.full(n, 1e27, np.float32)
        tmin[kind == 11] = -2.0
        tmax[kind == 12] = np.inf
        tmax[kind == 13] = 0.4
        tmin[kind == 14], tmax[kind == 14] = 1.0, 0.5
        tmin[kind == 15] = np.nan
        ot = torch.from_numpy(np.concatenate([o, tmin[:, None]], 1).astype(np.float32)).cuda()
        dt = torch.from_numpy(np.concatenate([d, tmax[:, None]], 1).astype(np.float32)).cuda()
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
        for a, b in zip(*got):
            assert np.array_equal(a, b)
        assert (got[0][0][kind == 0] >= 0).all()  # ordinary rays in a closed box
    R.close()
