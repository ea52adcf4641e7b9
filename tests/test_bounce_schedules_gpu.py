"""The wavefront's bounce schedules against one another with path pools off (small passes otherwise run by
pools, on which these options have no effect): overlapped and in order, one and two pipelines with several
chunks, every binning granularity, the 4-wide BVH, the BVH2 and the one-ray-per-thread kernels.  Every path's
arithmetic is its own, so images and counters are identical; the adjoint's gradients agree to the order
of their float sums."""
import numpy as np
import pytest

from open_rendering_framework_b200 import scene as sc
from open_rendering_framework_b200 import scenes

pytestmark = pytest.mark.gpu

COUNTS = ("path_samples", "segments", "shadow_rays", "clamped_indices", "capped_walks", "dipole_gathers", "dipole_pairs", "gather_overflows")


def render(make, frames, opts, max_paths=None):
    R = sc.Renderer(make(), max_paths_in_flight=max_paths)
    for k, v in opts.items():
        R.set_option(k, v)
    R.render(frames)
    R.render(frames)  # the second render reuses the streams, events and queues
    out = R.readback().view(np.uint32), [getattr(R.stats(), k) for k in COUNTS], R.stats().extend_launches
    R.close()
    return out


SCENES = {
    "single": lambda: scenes.single_scene(67, 45, 3, 2),
    "sky": lambda: scenes.env_scene(61, 40),
    "analytic_lights": lambda: scenes.analytic_light_scene(50, 41),
    "layered_multiple_scattering": lambda: scenes.layered_scene(53, 37, rough_model=sc.MULTISCATTERING_MODEL),
    "large": lambda: scenes.single_scene(256, 200, 4, 3),
}
ARMS = ({}, {"bin_items": 4}, {"bin_items": 16}, {"overlap": 0}, {"dual": 0}, {"dual": 0, "overlap": 0}, {"bvh4": 0}, {"extend_mode": 0}, {"refill": 31})


@pytest.mark.parametrize("name", list(SCENES))
def test_one_chunk(name):
    ref = render(SCENES[name], 3, {"pool": 2})
    for opts in ARMS:
        got = render(SCENES[name], 3, {"pool": 0, **opts})
        assert np.array_equal(ref[0], got[0]) and ref[1] == got[1], opts


@pytest.mark.parametrize("name", list(SCENES))
def test_two_pipelines_over_several_chunks(name):
    """Seven frames, two to a chunk: with dual 1 every chunk is one frame (seven chunks alternate between the
    pipelines), with dual 0 there are four chunks in turn."""
    make = SCENES[name]
    c = make().camera
    max_paths = 2 * c.width * c.height
    passes = make().integrator.max_depth + 2
    ref = render(make, 7, {"pool": 0, "dual": 0, "overlap": 0}, max_paths)
    assert ref[2] == 4 * passes
    for opts in ARMS:
        got = render(make, 7, {"pool": 0, **opts}, max_paths)
        assert np.array_equal(ref[0], got[0]) and ref[1] == got[1], opts
        assert got[2] == (4 if opts.get("dual") == 0 else 7) * passes
    pools = render(make, 7, {"pool": 2}, max_paths)
    assert np.array_equal(ref[0], pools[0]) and ref[1] == pools[1] and pools[2] == 7


@pytest.mark.parametrize("rough", [None, (0.25, sc.MULTISCATTERING_MODEL, sc.GGX_DISTRIBUTION)])
@pytest.mark.parametrize("max_paths", [None, 47 * 33])
def test_translucent_objects(rough, max_paths):
    make = lambda: scenes.translucent_box_scene(47, 33, probe_samples=1700, two_objects=True, rough=rough)  # noqa: E731
    ref = render(make, 3, {"pool": 0, "overlap": 0}, max_paths)
    for opts in ({"pool": 0}, {"pool": 0, "bin_items": 4}, {"pool": 0, "bvh4": 0}, {"pool": 2}, {"pool": 1}):
        got = render(make, 3, opts, max_paths)
        assert np.array_equal(ref[0], got[0]) and ref[1] == got[1], opts


@pytest.mark.parametrize("use_graph", [1, 0])
@pytest.mark.parametrize("max_paths", [None, 2000])
def test_batch(use_graph, max_paths):
    make = lambda: scenes.batch_scenes(6, seed=5, size_scale=0.1, spp_scale=0.05, env_w=64, env_h=32, probe_samples=40)  # noqa: E731
    items = make()
    ref = []
    for d, f, _ in items:
        R = sc.Renderer(d)
        R.set_option("pool", 0)
        R.set_option("overlap", 0)
        R.render(f)
        R.render(f)
        ref.append(R.readback().view(np.uint32))
        R.close()
    for opts in ({"pool": 0}, {"pool": 0, "overlap": 0}, {"pool": 0, "dual": 0}, {"pool": 2}):
        items = make()
        rs = [sc.Renderer(d) for d, _, _ in items]
        B = sc.Batch(rs, [f for _, f, _ in items])
        B.set_option("use_graph", use_graph)
        if max_paths:
            B.set_option("max_paths_in_flight", max_paths)
        for k, v in opts.items():
            B.set_option(k, v)
        B.render()
        B.render()
        for R, r in zip(rs, ref):
            assert np.array_equal(R.readback().view(np.uint32), r), opts
        B.close()
        for R in rs:
            R.close()


def test_adjoint_overlapped_and_in_order():
    torch = pytest.importorskip("torch")
    from open_rendering_framework_b200 import diff

    out = []
    for opts in ({"overlap": 1}, {"overlap": 0}, {"overlap": 1, "bin_items": 4}):
        data, (dif, met, tr) = scenes.inverse_scene(35, 29, subdiv=3, tex_res=30, probe_samples=64, seed=3)
        S = diff.DiffScene(data, dif, met, tr)
        S.R.set_option("pool", 0)
        for k, v in opts.items():
            S.R.set_option(k, v)
        p = [torch.from_numpy(x.copy()).cuda().requires_grad_() for x in
             (dif.texture, met.texture, np.r_[np.asarray(tr.absorption, np.float32), np.asarray(tr.scattering, np.float32)])]
        img = diff.render(S, 3, *p)
        out.append([img.detach()] + list(torch.autograd.grad((img ** 2).sum(), p)))
        S.close()
    for other in out[1:]:
        assert torch.equal(out[0][0], other[0])
        for a, b in zip(out[0][1:], other[1:]):
            # sums of up to some thousand float terms in another order
            assert float((a - b).double().norm()) <= 5e-5 * float(a.double().norm()) and float(a.norm()) > 0
