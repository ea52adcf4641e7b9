"""Dipole gathers at the edges of the gather kernel: probe counts around a warp's queue (32 pairs per
evaluation), acceptance from nearly every pair (the queue fills at every step) to nearly none, one and
two translucent objects (lanes of one warp then hold gathers of different sets), and patches that leave
a warp with a single path.  Against the oracle's sequential gathers, with the image bars of the
translucent renders (95% of the pixels within 1e-3 relative, relative MSE below 1e-4)."""
import numpy as np
import pytest

from oracle import oracle_ctypes as oc
from open_rendering_framework_b200 import scene as sc
from open_rendering_framework_b200 import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("probes,scale,model,two,size", [
    (1, 10.0, sc.STANDARD_DIPOLE, False, 24), (31, 1.0, sc.STANDARD_DIPOLE, False, 24), (33, 1.0, sc.DIRECTIONAL_DIPOLE, True, 24),
    (130, 400.0, sc.STANDARD_DIPOLE, True, 24), (257, 40.0, sc.DIRECTIONAL_DIPOLE, False, 24), (64, 4.0, sc.STANDARD_DIPOLE, True, 3)])
def test_gathers_at_queue_edges_match_oracle(probes, scale, model, two, size):
    data = scenes.translucent_box_scene(size, size, subdiv=2, probe_samples=probes, dipole_model=model, two_objects=two)
    for m in data.materials:
        if isinstance(m, sc.TranslucentMaterial):
            m.setScale(scale)
    R = sc.Renderer(data)
    R.render(3)
    got, st = R.readback(), R.stats()
    R.close()
    O = oc.OracleScene(data)
    ref, _ = O.render(0, 3, accum=np.zeros((size, size, 4), np.float32), threads=8)
    O.close()
    assert st.gather_overflows == 0 and np.all(np.isfinite(got))
    g, r = got[..., :3].astype(np.float64), ref[..., :3].astype(np.float64)
    ok = np.mean(np.all(np.abs(g - r) <= 1e-3 * np.maximum(np.abs(r), 1e-3), axis=-1))
    mse = np.mean((g - r) ** 2) / max(np.mean(r ** 2), 1e-30)
    assert ok >= 0.95 and mse < 1e-4, (ok, mse)
    assert st.dipole_gathers > 0 or size < 8
