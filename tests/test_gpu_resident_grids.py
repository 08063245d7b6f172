"""Energy passes and force gathers whose grids hold no more blocks than the chip does and stride over their items: cloths
with springs just below, at and beyond one round of 152 SMs x 2,048 threads (311,296), against the oracle.  Energies and
forces of plain FP64 within 1e-10 relative (sums of at most 1.9M positive terms and of 12 spring forces a vertex).
"""
import numpy as np
import pytest

from oracle import scenes as oscenes
from ssim_gb300 import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [225, 229, 300, 560])
def test_cloth_energy_and_forces(n):
    sc = scenes.cloth(n, h=0.05, k=1e3, areal_density=0.5, dt=1e-2)
    ts, ot = scenes.build_timestep(sc, stepper="none"), oscenes.build_oracle(sc)
    u = np.random.default_rng(n).uniform(-1, 1, sc["X"].shape) * 0.02
    for t in (ts, ot):
        t.prepare_step()
        t.set("next_deform", u)
    e, eo = ts.update_energy_and_gradients(), ot.update_energy_and_gradients()
    f, fo = ts.get("forces"), ot.get("forces")
    assert abs(e - eo) <= 1e-10 * abs(eo)
    assert np.abs(f - fo).max() <= 1e-10 * np.abs(fo).max()
    assert abs(ts.energy_at(0.5 * u) - ot.energy_at(0.5 * u)) <= 1e-10 * abs(eo)
