"""The resident FP64 PCG (kernels_pcg.cu) where it is reached: its own layouts, tuned handles, scales of the right side."""
import numpy as np
import pytest

import ssim_gb300 as g
from ssim_gb300 import mesh

pytestmark = pytest.mark.gpu


def _handle(hexes, tune=None, **params):
    X, T = mesh.kuhn_box(hexes, tuple(0.1 * k for k in hexes))
    X = mesh.jitter_interior(X, 0.008, 71)
    fixed = np.where(X[:, 0] == 0.0)[0]
    ts = g.TimeStep(X, T, 1e-2, 1e5, 0.45, 1000.0)
    ts.set_precision("fp64")
    ts.set_material(10.0 ** mesh.uniform(72, T.shape[0], 4.0, 6.0), None)
    ts.mark_dirichlet_batched(fixed, np.zeros((fixed.size, 3)))
    ts.set_params(g.default_params(precond=2, cg_max_iters=20000, **params))
    ts.reset("newton")
    if tune is not None:
        tune(ts)
    ts.update_hessian(False, True, True)
    return ts, np.random.default_rng(73).normal(size=X.shape)


def test_tuned_handle_solves_on_chip():
    """autotune() and set_tuning() keep the automatic choice's solve: the bits of an untuned handle's.  A variant asked
    for afterwards outranks the tuning, by change or by name; other parameters leave it."""
    ref, b = _handle((13, 9, 7))
    x, it, rr = ref.pcg(b, rtol=1e-6)
    ref.set_params(pcg_persistent=0)
    x0, _, _ = ref.pcg(b, rtol=1e-6)
    assert not np.array_equal(x, x0)
    saved = {}
    ts, _ = _handle((13, 9, 7), tune=lambda t: saved.update(t.autotune()))
    ts2, _ = _handle((13, 9, 7), tune=lambda t: t.set_tuning(saved))
    assert saved["pcg_solve_ms"] > 0 and saved["pcg_iterations"] > 0
    for t in (ts, ts2):
        t.set_params(cg_check_every=8)
        got = t.pcg(b, rtol=1e-6)
        assert np.array_equal(got[0], x) and got[1:] == (it, rr)
        for variant in (0, 2, 0):
            t.set_params(pcg_persistent=variant)
            assert np.array_equal(t.pcg(b, rtol=1e-6)[0], x0) == (variant == 0)


@pytest.mark.parametrize("hexes", [(13, 9, 7), (24, 24, 24)])
def test_solutions_scale_with_the_right_side(hexes):
    """A right side times a power of two gives the solution times it, bit for bit: nothing in the iteration leaves FP64's
    range while the residual's square is inside it."""
    ts, b = _handle(hexes)
    for rtol in (5e-2, 1e-8):
        x, it, rr = ts.pcg(b, rtol=rtol)
        for k in (-400, -280, 280, 400):
            got = ts.pcg(np.ldexp(b, k), rtol=rtol)
            assert got[1:] == (it, rr) and np.array_equal(np.ldexp(got[0], -k), x), (rtol, k, got[1:], (it, rr))


def test_solves_that_do_not_fit_take_no_scratch():
    """132,651 vertices are beyond the chip (25 slices on each of 152 SMs): the automatic choice runs the two-launch loop,
    bit for bit, and does not allocate the resident solve's vectors (8.5 MB; the driver hands out 2 MB at a time)."""
    import torch

    ts, b = _handle((50, 50, 50))
    ts.set_params(pcg_persistent=0)
    x0, it0, _ = ts.pcg(b, rtol=5e-2)
    free = torch.cuda.mem_get_info()[0]
    ts.set_params(pcg_persistent=3)
    x, it, _ = ts.pcg(b, rtol=5e-2)
    assert it == it0 and np.array_equal(x, x0)
    assert free - torch.cuda.mem_get_info()[0] <= 4 << 20
