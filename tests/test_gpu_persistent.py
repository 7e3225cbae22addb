"""The persistent on-chip CG kernel against the batched sweeps (TL_CG_PERSISTENT=0) after a few
iterations, field by field, at the sizes where its tilings change: one CTA, one cluster (its last
CTAs without a tile), the whole grid; one to eighteen cells a thread; meshes one cell wide or high;
ragged last tiles; the largest mesh that fits.

Both forms do the same arithmetic per cell and differ in the rounding of the sums p.w and r.z only:
alpha and beta agree to a few units of 2^-53, so after N iterations a field differs by at most some
N times 2^-52 of its largest value, times the growth of a perturbation along the iteration, below
1e3 for the few iterations taken here: 1e-11 holds for all fields."""
import numpy as np
import pytest

from helpers import small_deck

pytestmark = pytest.mark.gpu

SIZES = [(2, 2), (10, 10), (21, 22), (1, 900), (900, 1), (33, 31), (61, 60), (105, 104), (127, 129), (1, 20000),
         (20000, 3), (256, 256), (301, 499), (512, 512), (700, 641), (777, 1013), (1000, 1000), (1099, 1097)]


@pytest.mark.parametrize("case", [dict(), dict(precond="jac_diag", reflective=True)], ids=["none", "diag-reflective"])
@pytest.mark.parametrize("size", SIZES, ids=["%dx%d" % s for s in SIZES])
def test_persistent_iterations_match_the_sweeps(size, case, monkeypatch):
    from tealeaf_ref_gb300 import native

    fields = ["u", "r", "p", "w"] + (["z"] if "precond" in case else [])
    d = small_deck(nx=size[0], ny=size[1], steps=1, n_rect=4, n_circ=2, max_iters=9, **case)
    if size == (2, 2):
        d.max_iters = 1
    runs = []
    for form in ("0", "1"):
        monkeypatch.setenv("TL_CG_PERSISTENT", form)
        with native.Chunk.from_deck(d) as c:
            i = c.tea_leaf(d)
            runs.append((i, {f: c.download(f) for f in fields}))
    (i0, f0), (i1, f1) = runs
    assert i1.kernel_launches < i0.kernel_launches, "the persistent kernel did not run"
    assert i1.n_exit == i0.n_exit and i1.cg_calc_steps == i0.cg_calc_steps
    assert abs(i1.error - i0.error) <= 1e-11 * i0.initial_residual
    for f in fields:
        assert np.max(np.abs(f1[f] - f0[f])) <= 1e-11 * np.max(np.abs(f0[f])), f


MIXED_SIZES = [(20, 20), (1, 3000), (3000, 1), (301, 199), (511, 513), (1000, 1000), (1499, 1999), (2048, 2048)]


@pytest.mark.parametrize("case", [dict(), dict(precond="jac_diag", reflective=True)], ids=["none", "diag-reflective"])
@pytest.mark.parametrize("size", MIXED_SIZES, ids=["%dx%d" % s for s in MIXED_SIZES])
def test_persistent_fp32_steps_match_the_sweeps(size, case, monkeypatch):
    """The precision form capped at 8 FP32 steps and the replacement that follows.  Both forms do the
    same FP32 arithmetic per cell; the sums' rounding can move alpha and beta, as floats, by one
    unit (2^-23) a step, so the correction u - u0 agrees to 8 steps x 2 x 2^-23, times 8 for the
    growth of a perturbation along them."""
    from tealeaf_ref_gb300 import native

    d = small_deck(nx=size[0], ny=size[1], steps=1, n_rect=4, n_circ=2, **case)
    o = native.opts_from_deck(d, "mixed", inner_tol=1e-6, max_inner_iters=8)
    runs = []
    for form in ("0", "1"):
        monkeypatch.setenv("TL_CG_PERSISTENT", form)
        with native.Chunk.from_deck(d) as c:
            i = c.tea_leaf(o, d.initial_timestep)
            runs.append((i, c.download("u"), c.download("u0")))
    (i0, u0, b), (i1, u1, _) = runs
    assert i1.kernel_launches < i0.kernel_launches, "the persistent kernel did not run"
    assert i1.cg_calc_steps == i0.cg_calc_steps == 8 and i1.outer_iterations == i0.outer_iterations
    assert np.max(np.abs(u1 - u0)) <= 8 * 2 * 8 * 2.0 ** -23 * np.max(np.abs(u0 - b))
