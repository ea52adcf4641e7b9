"""Path pools (option "pool" = 2, every bounce of a pass in one launch) against the wavefront's launches
(option 0): every path runs the same functions on the same records, so the images and the counters are
identical.  Sizes: a single pixel, fewer paths than a warp, ragged sizes, a patch that leaves most pixels
out, and more paths than all pools hold at once (blocks then take new paths while others continue);
programs: basic, translucent, and all (layered, multiple scattering, rough translucent); many scenes in
one pass; and the adjoint's gradients, which the two schedules add up in another order (5e-5 relative: a
texel's sum of up to some thousand float terms)."""
import numpy as np
import pytest

from open_rendering_framework_b200 import scene as sc
from open_rendering_framework_b200 import scenes

pytestmark = pytest.mark.gpu

COUNTS = ("path_samples", "segments", "shadow_rays", "clamped_indices", "capped_walks", "dipole_gathers", "dipole_pairs", "gather_overflows")


def render(data, frames, pool):
    R = sc.Renderer(data)
    R.set_option("pool", pool)
    R.render(frames)
    img, st = R.readback(), R.stats()
    R.close()
    return img, [getattr(st, k) for k in COUNTS]


def patch(data):
    data.camera.patch_origin, data.camera.patch_dims = (3, 2), (5, 4)
    return data


SCENES = {
    "one_pixel": (lambda: scenes.single_scene(1, 1, 2, 2), 1),
    "few_paths": (lambda: scenes.single_scene(5, 3, 3, 2), 1),
    "ragged": (lambda: scenes.single_scene(67, 45, 3, 2), 3),
    "patch": (lambda: patch(scenes.single_scene(33, 31, 3, 2)), 2),
    "more_than_the_pools_hold": (lambda: scenes.single_scene(512, 512, 3, 2), 5),
    "sky": (lambda: scenes.env_scene(61, 40), 2),
    "analytic_lights": (lambda: scenes.analytic_light_scene(50, 41), 2),
    "layered_multiple_scattering": (lambda: scenes.layered_scene(53, 37, rough_model=sc.MULTISCATTERING_MODEL), 2),
    "multiple_scattering": (lambda: scenes.single_scene(53, 37, 3, 2, metal_model=sc.MULTISCATTERING_MODEL, glass_model=sc.MULTISCATTERING_MODEL), 2),
    "translucent": (lambda: scenes.translucent_box_scene(47, 33, probe_samples=70, two_objects=True), 2),
    "rough_translucent": (lambda: scenes.translucent_box_scene(41, 33, probe_samples=70, rough=(0.25, sc.MULTISCATTERING_MODEL, sc.GGX_DISTRIBUTION)), 2),
}


@pytest.mark.parametrize("name", list(SCENES))
def test_pools_match_the_wavefront(name):
    make, frames = SCENES[name]
    a, ca = render(make(), frames, 0)
    b, cb = render(make(), frames, 2)
    assert np.array_equal(a.view(np.uint32), b.view(np.uint32)) and ca == cb


def test_pools_match_the_wavefront_in_a_batch():
    images = []
    for pool in (0, 2):
        items = scenes.batch_scenes(6, seed=5, size_scale=0.1, spp_scale=0.05, env_w=64, env_h=32, probe_samples=40)
        rs = [sc.Renderer(d) for d, _, _ in items]
        B = sc.Batch(rs, [f for _, f, _ in items])
        B.set_option("pool", pool)
        B.render()
        B.render()
        images.append([R.readback() for R in rs])
        B.close()
        for R in rs:
            R.close()
    assert all(np.array_equal(a.view(np.uint32), b.view(np.uint32)) for a, b in zip(*images))


def test_pools_adjoint_matches_the_wavefront():
    torch = pytest.importorskip("torch")
    from open_rendering_framework_b200 import diff

    grads = []
    for pool in (0, 2):
        data, (dif, met, tr) = scenes.inverse_scene(35, 29, subdiv=3, tex_res=30, probe_samples=64, seed=3)
        S = diff.DiffScene(data, dif, met, tr)
        S.R.set_option("pool", pool)
        p = [torch.from_numpy(x.copy()).cuda().requires_grad_() for x in
             (dif.texture, met.texture, np.r_[np.asarray(tr.absorption, np.float32), np.asarray(tr.scattering, np.float32)])]
        img = diff.render(S, 3, *p)
        grads.append([img.detach()] + list(torch.autograd.grad((img ** 2).sum(), p)))
        S.close()
    assert torch.equal(grads[0][0], grads[1][0])
    for a, b in zip(grads[0][1:], grads[1][1:]):
        assert float((a - b).double().norm()) <= 5e-5 * float(a.double().norm()) and float(a.norm()) > 0


@pytest.mark.parametrize("value", [-1, 3])
def test_pool_option_rejects_other_values(value):
    R = sc.Renderer(scenes.single_scene(4, 4, 1, 1))
    with pytest.raises(Exception):
        R.set_option("pool", value)
    R.close()


@pytest.mark.parametrize("probes,frames", [(1, 1), (70, 3), (3000, 2)])
def test_probe_paths_beside_the_camera_paths(probes, frames):
    """The probe pass on its own stream and wavefront (option overlap 1, pools) against the one after the other
    (overlap 0) and the wavefront's launches (pool 0): images, counters and probe records are identical, over
    two renders of one context."""
    got = []
    for pool, overlap in ((1, 1), (1, 0), (0, 1)):
        R = sc.Renderer(scenes.translucent_box_scene(40, 31, probe_samples=probes, two_objects=True))
        R.set_option("pool", pool)
        R.set_option("overlap", overlap)
        R.render(frames)
        first = [getattr(R.stats(), k) for k in COUNTS]
        R.render(frames)
        got.append((R.readback().view(np.uint32), first, [getattr(R.stats(), k) for k in COUNTS], R.probes().tobytes()))
        R.close()
    for other in got[1:]:
        assert np.array_equal(got[0][0], other[0]) and got[0][1:] == other[1:]
