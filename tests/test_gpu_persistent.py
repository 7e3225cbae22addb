"""The loops on chip against the sweeps in memory.  The CG kernels (TL_CG_PERSISTENT=0 forces the
batched sweeps) after a few iterations, field by field, at the sizes where their tilings change: one
CTA, one cluster (its last CTAs without a tile), the whole grid; one to eleven cells a thread, and
the form of larger tiles; meshes one cell wide or high; ragged last tiles; nearly the largest mesh
that fits.

Both forms do the same arithmetic per cell and differ in the rounding of the sums p.w and r.z only:
alpha and beta agree to a few units of 2^-53, so after N iterations a field differs by at most some
N times 2^-52 of its largest value, times the growth of a perturbation along the iteration, below
1e3 for the few iterations taken here: 1e-11 holds for all fields."""
import numpy as np
import pytest

from helpers import small_deck

pytestmark = pytest.mark.gpu

SIZES = [(2, 2), (10, 10), (21, 22), (1, 900), (900, 1), (33, 31), (61, 60), (105, 104), (127, 129), (1, 20000),
         (20000, 3), (256, 256), (301, 499), (512, 512), (700, 641), (777, 1013), (1000, 1000), (1099, 1097),
         (1391, 1399)]


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


MIXED_SIZES = [(20, 20), (1, 3000), (3000, 1), (1, 40000), (40000, 1), (301, 199), (511, 513), (701, 699), (745, 753),
               (1000, 1000), (2047, 1021), (1499, 1999), (2048, 2048)]


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


POLY_SIZES = [(9, 9), (22, 21), (1, 700), (700, 1), (97, 131), (301, 499), (600, 433), (777, 813), (1000, 1000), (1003, 1201),
              (1399, 1391)]


@pytest.mark.parametrize("precond", ["none", "jac_diag"])
@pytest.mark.parametrize("solver", ["ppcg", "chebyshev"])
@pytest.mark.parametrize("size", POLY_SIZES, ids=["%dx%d" % s for s in POLY_SIZES])
def test_on_chip_polynomial_steps_give_the_same_bits(size, solver, precond, monkeypatch):
    """The FP64 PPCG inner steps and Chebyshev iterations on chip against the sweeps in memory: the
    same bits in every field, over two time steps (with odd and even step counts, and residual checks
    between launches)."""
    from tealeaf_ref_gb300 import native

    d = small_deck(nx=size[0], ny=size[1], solver=solver, precond=precond, ppcg_inner_steps=7, ch_cg_presteps=6,
                   ch_cg_epslim=1e30, max_iters=14 if solver == "ppcg" else 87, steps=2)
    fields = ["u", "w", "r", "p", "sd", "rtemp", "utemp"] + (["z"] if precond == "jac_diag" else [])
    runs = []
    for form in ("0", "1"):
        monkeypatch.setenv("TL_POLY_PERSISTENT", form)
        with native.Chunk.from_deck(d) as c:
            infos = [c.tea_leaf(d) for _ in range(2)]
            runs.append((infos, {f: c.download(f) for f in fields}))
    (i0, f0), (i1, f1) = runs
    assert sum(i.cheby_calc_steps for i in i0) > 0
    assert sum(i.kernel_launches for i in i1) < sum(i.kernel_launches for i in i0), "the on-chip steps did not run"
    for a, b in zip(i0, i1):
        assert (a.n_exit, a.error, a.cheby_calc_steps, a.ppcg_inner_iters) == \
               (b.n_exit, b.error, b.cheby_calc_steps, b.ppcg_inner_iters)
    for f in fields:
        assert np.array_equal(f0[f], f1[f]), f


@pytest.mark.parametrize("solver", ["ppcg", "chebyshev"])
def test_on_chip_polynomial_wait_is_bounded(solver, monkeypatch):
    """One tile keeps its rim to itself: its neighbours' waits run out after about a second, the solve
    returns TL_ERR_TIMEOUT, and the context then solves normally."""
    from tealeaf_ref_gb300 import native

    d = small_deck(nx=200, ny=160, solver=solver, ppcg_inner_steps=6, ch_cg_presteps=10, ch_cg_epslim=1e30,
                   max_iters=60, steps=1)
    with native.Chunk.from_deck(d) as c:
        want = c.tea_leaf(d)
        c.generate(d)
        c.reset_eigen()
        monkeypatch.setenv("TL_CG_BARRIER_EXTRA", "2")
        with pytest.raises(native.TeaLeafError) as e:
            c.tea_leaf(d)
        assert e.value.code == -5  # TL_ERR_TIMEOUT
        monkeypatch.delenv("TL_CG_BARRIER_EXTRA")
        c.generate(d)
        c.reset_eigen()
        got = c.tea_leaf(d)
        assert (got.n_exit, got.error) == (want.n_exit, want.error)


MIXED_POLY_SIZES = [(9, 9), (1, 700), (700, 1), (97, 131), (301, 499), (640, 613), (999, 1001), (1499, 1999), (2039, 2043)]


@pytest.mark.parametrize("case", [dict(), dict(precond="jac_diag", reflective=True)], ids=["none", "diag-reflective"])
@pytest.mark.parametrize("solver", ["ppcg", "chebyshev"])
@pytest.mark.parametrize("size", MIXED_POLY_SIZES, ids=["%dx%d" % s for s in MIXED_POLY_SIZES])
def test_on_chip_fp32_polynomial_steps_give_the_same_bits(size, solver, case, monkeypatch):
    """The FP32 PPCG inner steps and Chebyshev cycles of the precision form on chip against the blocked
    sweeps: the same bits in every FP64 field."""
    from tealeaf_ref_gb300 import native

    d = small_deck(nx=size[0], ny=size[1], solver=solver, ppcg_inner_steps=7, ch_cg_presteps=6, ch_cg_epslim=1e30,
                   max_iters=14 if solver == "ppcg" else 87, steps=1, **case)
    o = native.opts_from_deck(d, "mixed")
    fields = ["u", "r", "p"] + (["w", "z"] if solver == "ppcg" else [])
    runs = []
    for form in ("0", "1"):
        monkeypatch.setenv("TL_POLY_PERSISTENT", form)
        with native.Chunk.from_deck(d) as c:
            i = c.tea_leaf(o, d.initial_timestep)
            runs.append((i, {f: c.download(f) for f in fields}))
    (i0, f0), (i1, f1) = runs
    assert i0.cheby_calc_steps > 0
    assert i1.kernel_launches < i0.kernel_launches, "the on-chip steps did not run"
    assert (i0.n_exit, i0.error, i0.cheby_calc_steps, i0.ppcg_inner_iters) == \
           (i1.n_exit, i1.error, i1.cheby_calc_steps, i1.ppcg_inner_iters)
    for f in fields:
        assert np.array_equal(f0[f], f1[f]), f


@pytest.mark.parametrize("solver", ["ppcg", "chebyshev"])
def test_on_chip_fp32_polynomial_wait_is_bounded(solver, monkeypatch):
    """As test_on_chip_polynomial_wait_is_bounded, for the precision form."""
    from tealeaf_ref_gb300 import native

    d = small_deck(nx=200, ny=160, solver=solver, ppcg_inner_steps=6, ch_cg_presteps=10, ch_cg_epslim=1e30,
                   max_iters=60, steps=1)
    o = native.opts_from_deck(d, "mixed")
    with native.Chunk.from_deck(d) as c:
        want = c.tea_leaf(o, d.initial_timestep)
        c.generate(d)
        c.reset_eigen()
        monkeypatch.setenv("TL_CG_BARRIER_EXTRA", "2")
        with pytest.raises(native.TeaLeafError) as e:
            c.tea_leaf(o, d.initial_timestep)
        assert e.value.code == -5  # TL_ERR_TIMEOUT
        monkeypatch.delenv("TL_CG_BARRIER_EXTRA")
        c.generate(d)
        c.reset_eigen()
        got = c.tea_leaf(o, d.initial_timestep)
        assert (got.n_exit, got.error) == (want.n_exit, want.error)


def test_on_chip_solves_of_two_threads():
    """Two threads, each with chunks of its own, solve at the same time in every on-chip form: the bits
    are those of the same solves one after the other."""
    import threading

    from tealeaf_ref_gb300 import native

    work = [(solver, precision, size) for size in ((200, 160), (420, 390))
            for solver, precision in (("cg", "fp64"), ("cg", "mixed"), ("ppcg", "fp64"), ("ppcg", "mixed"),
                                      ("chebyshev", "mixed"))]

    def solve_all(order, out):
        for k in order:
            solver, precision, (nx, ny) = work[k]
            d = small_deck(nx=nx, ny=ny, solver=solver, ch_cg_presteps=10, ch_cg_epslim=1e30, ppcg_inner_steps=6,
                           max_iters=120, steps=1)
            with native.Chunk.from_deck(d) as c:
                c.tea_leaf(native.opts_from_deck(d, precision), d.initial_timestep)
                out[k] = c.download("u")

    want, got = {}, [{}, {}]
    solve_all(range(len(work)), want)
    orders = [range(len(work)), range(len(work) - 1, -1, -1)]
    threads = [threading.Thread(target=solve_all, args=(o, g)) for o, g in zip(orders, got)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for g in got:
        for k in range(len(work)):
            assert k in g and np.array_equal(g[k], want[k]), work[k]
