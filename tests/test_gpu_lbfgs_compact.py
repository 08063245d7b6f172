"""The compact L-BFGS direction (kernels_lbfgs.cu) against the two-loop recursion: eight pairs fit the compact form, nine
do not, and within eight iterations both keep the same pairs, so steps capped at eight iterations agree up to rounding.
FP64 to 1e-9 (1e-16 amplified by the line search's decisions never, by eight iterations of H g by their conditioning).
Sizes on both sides of the two multidot layouts' border (19,456 vertices on 152 SMs) and a mesh smaller than a block."""
import numpy as np
import pytest

import ssim_gb300 as g
from ssim_gb300 import mesh

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("hexes", [(2, 2, 2), (12, 7, 5), (30, 25, 23), (30, 25, 24)])
def test_compact_matches_two_loop(hexes):
    X, T = mesh.kuhn_box(hexes, tuple(0.05 * k for k in hexes))
    X = mesh.jitter_interior(X, 0.004, 41)
    fixed = np.where(X[:, 0] == 0.0)[0]
    v0 = 0.2 * np.random.default_rng(42).normal(size=X.shape)
    out = []
    for history in (8, 9):
        ts = g.TimeStep(X, T, 1e-2, 1e5, 0.4, 1000.0)
        ts.mark_dirichlet_batched(fixed, np.zeros((fixed.size, 3)))
        ts.set_params(g.default_params(stop_mode=1, rel_tol=1e-12, lbfgs_history=history, max_lbfgs_iters=8))
        ts.reset("lbfgs")
        ts.set("velocity", v0)
        ts.step()
        assert ts.stats()["newton_iters"] == 8
        out.append(ts.get("deformation"))
    assert np.linalg.norm(out[0] - out[1]) <= 1e-9 * np.linalg.norm(out[1])
