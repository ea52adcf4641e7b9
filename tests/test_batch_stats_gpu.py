"""Statistics of a batch render that replays its graph after another pass has run on the engine."""
import pytest

from open_rendering_framework_b200 import scene as sc
from open_rendering_framework_b200 import scenes

pytestmark = pytest.mark.gpu

COUNTS = ("path_samples", "segments", "shadow_rays", "dipole_gathers", "dipole_pairs")


@pytest.mark.parametrize("first,max_paths", [
    (lambda: scenes.translucent_box_scene(40, 31, probe_samples=500), None),  # probe paths counted beside
    (lambda: scenes.single_scene(64, 64, 3, 2), 16384),                       # two pipelines, each with its counts
])
def test_replay_after_a_sequential_render_counts_every_path(first, max_paths):
    rs = [sc.Renderer(first()), sc.Renderer(scenes.single_scene(16, 16, 2, 2))]
    B = sc.Batch(rs, [4, 1])
    if max_paths:
        B.set_option("max_paths_in_flight", max_paths)
    got = []
    for sequential in (False, True, False):  # the second batched render replays the first one's graph
        for R in rs:
            R.apply_camera()  # the images start over, so that every render traces the same frames
        if sequential:
            B.render_sequential()
        else:
            B.render()
            st = B.stats()
            got.append([getattr(st, k) for k in COUNTS])
    B.close()
    for R in rs:
        R.close()
    assert got[0] == got[1] and got[0][1] > got[0][0]
