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


# hexes a side, grid cap, whether the vectors fit on chip
LAYOUTS = [
    ((13, 9, 7), 18, True),    # 35 slices, two a block: four warps a slice, entries on chip
    ((13, 9, 7), 12, True),    # three a block
    ((7, 7, 7), 4, True),      # 16 slices, four a block: two warps a slice, entries on chip
    ((24, 24, 24), 0, True),   # 489 slices, three and four a block
    ((13, 9, 7), 7, True),     # five a block, entries in global memory
    ((15, 9, 9), 2, True),     # 50 slices, 25 a block: the most whose vectors fit
    ((15, 12, 7), 2, False),   # 52 slices, 26 a block: the two-launch loop
]


@pytest.mark.parametrize("hexes,blocks,fits", LAYOUTS)
def test_solve_matches_two_launch_in_its_layouts(hexes, blocks, fits):
    """Against the two-launch loop, in the layouts of the FP64 kernel, with the path that ran read from the profile:
    iteration counts within 2, true residuals at 1.5 of the tolerance, a capped solve's iterate within 1e-12."""
    ts, b = _handle(hexes, pcg_max_blocks=blocks)
    bn = np.linalg.norm(b)
    for rtol in (5e-2, 1e-6, 1e-10):
        ts.set_params(pcg_persistent=3)
        ts.profile(True)
        x, it, rr = ts.pcg(b, rtol=rtol)
        one, two = (ts.profile_read(k)["launches"] for k in ("pcg_iteration", "pcg_spmv"))
        ts.profile(False)
        assert (one, two) == ((it, 0) if fits else (0, it))
        ts.set_params(pcg_persistent=0)
        _, it0, _ = ts.pcg(b, rtol=rtol)
        assert rr <= rtol and abs(it - it0) <= 2, (rtol, it, it0)
        assert np.linalg.norm(b - ts.spmv(x)) <= 1.5 * rtol * bn
    for rtol, pipe in ((1e-2, 80), (1e-2, 3), (1e-12, 80)):
        ts.set_params(pcg_persistent=3, pcg_pipe_iters=pipe)
        x, it, _ = ts.pcg(b, rtol=rtol, max_iters=7)
        ts.set_params(pcg_persistent=0)
        x0, it0, _ = ts.pcg(b, rtol=rtol, max_iters=7)
        assert it == it0 and np.linalg.norm(x - x0) <= 1e-12 * np.linalg.norm(x0)
