"""The batch autotuner times the schedule that the batch's full render takes: the wavefront's launches for a
render above the path pools' line, however few frames a trial has, and no search of the binning's
granularity where the full render runs by pools."""
import pytest

from open_rendering_framework_b200 import scene as sc
from open_rendering_framework_b200 import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("frames,pools", [(60, False), (4, True)])  # 1.97 M and 131 K paths; the line is at 1.57 M
def test_trials_run_on_the_schedule_of_the_full_render(frames, pools):
    rs = [sc.Renderer(scenes.single_scene(128, 128, 3, 2)) for _ in range(2)]
    B = sc.Batch(rs, [frames, frames])
    tuned = B.autotune(frames_per_trial=1)
    last = B.stats().kernel_launches  # of the last trial
    assert tuned.trials == (10 if pools else 12)  # ten settings of the traversal, then two granularities
    if not pools:
        assert last > 60
    B.render()
    n = B.stats().kernel_launches
    assert (n < 10) == (pools and tuned.extend_mode == 1), n
    B.close()
    for R in rs:
        R.close()
