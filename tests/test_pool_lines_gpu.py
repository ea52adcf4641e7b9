"""Where a batch's pass goes over from path pools to the wavefront's launches (a chunk by pools takes at most
nine launches, one by the wavefront more than eleven a bounce): passes of several scenes with translucent
objects, with the smooth program alone and with every program, below and above their lines."""
import pytest

from open_rendering_framework_b200 import scene as sc
from open_rendering_framework_b200 import scenes

pytestmark = pytest.mark.gpu

ROUGH = (0.25, sc.MULTISCATTERING_MODEL, sc.GGX_DISTRIBUTION)
KINDS = {
    "smooth": lambda: scenes.translucent_box_scene(128, 128, probe_samples=20),
    "rough": lambda: scenes.translucent_box_scene(128, 128, probe_samples=20, rough=ROUGH),
    "layered": lambda: scenes.layered_scene(128, 128, 2, rough_model=sc.MULTISCATTERING_MODEL),
}


@pytest.mark.parametrize("kinds,frames,pools", [
    (("smooth", "smooth"), 60, True), (("smooth", "smooth"), 70, True),  # 1.97 M and 2.29 M paths, line at 2^23
    (("rough", "rough"), 60, True), (("rough", "rough"), 70, False),     # line at 2^21
    (("smooth", "layered"), 60, True), (("smooth", "layered"), 70, False),
])
def test_line_of_translucent_passes_of_several_scenes(kinds, frames, pools):
    rs = [sc.Renderer(KINDS[k]()) for k in kinds]
    B = sc.Batch(rs, [frames] * len(rs))
    B.render()
    n = B.stats().kernel_launches
    B.close()
    for R in rs:
        R.close()
    assert (n <= 9) == pools, n
