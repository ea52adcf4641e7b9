"""The probe paths that run beside the camera paths: what their wavefront holds, and when it is used."""
import pytest

from open_rendering_framework_b200 import scene as sc
from open_rendering_framework_b200 import scenes

pytestmark = pytest.mark.gpu


def test_probe_wavefront_holds_only_what_pools_read():
    """A first render with the probe pass on its own wavefront (option overlap 1) takes at most the 150 bytes a
    probe path that the pools read, and 4 MB of granularity, more than one without (overlap 0)."""
    torch = pytest.importorskip("torch")
    probes = 200_000
    used = []
    for overlap in (0, 0, 1):  # the first round brings in the kernels' own memory
        R = sc.Renderer(scenes.translucent_box_scene(16, 16, probe_samples=probes))
        R.set_option("overlap", overlap)
        before = torch.cuda.mem_get_info()[0]
        R.render(1)
        R.sync()
        used.append(before - torch.cuda.mem_get_info()[0])
        R.close()
    assert 100 * probes < used[2] - used[1] <= 150 * probes + (4 << 20), used


@pytest.mark.parametrize("max_paths,beside", [(40 * 31, False), (40 * 31 + 5999, False), (40 * 31 + 6000, True)])
def test_probe_paths_keep_to_the_bound_on_paths_in_flight(max_paths, beside):
    """One frame of 1,240 camera paths and 6,000 probe paths: beside one another only where max_paths_in_flight
    holds both, else one after the other (the launches of option overlap 0)."""
    launches = []
    for overlap in (1, 0):
        R = sc.Renderer(scenes.translucent_box_scene(40, 31, probe_samples=3000, two_objects=True), max_paths_in_flight=max_paths)
        R.set_option("overlap", overlap)
        R.render(1)  # uploads and normals
        R.render(1)
        launches.append(R.stats().kernel_launches)
        R.close()
    in_order = 3 * -(-6000 // (40 * 31)) + 1 + 5  # generate, trace, finish per 1,240 probes; compact; the camera paths
    assert launches == [9 if beside else in_order, in_order], launches


def test_launches_that_trace_paths_are_counted_beside_and_in_order():
    """extend_launches counts a pool launch for the probe paths and one for the camera paths, on either stream."""
    got = []
    for overlap in (1, 0):
        R = sc.Renderer(scenes.translucent_box_scene(40, 31, probe_samples=200))
        R.set_option("overlap", overlap)
        R.render(2)
        got.append(R.stats().extend_launches)
        R.close()
    assert got == [2, 2]
