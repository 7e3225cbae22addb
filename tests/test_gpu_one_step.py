"""A single polynomial step runs as a sweep in memory, also on meshes whose steps run on chip: a tile on
chip reads its neighbours' cells from the field it overwrites at the end, and with one step nothing
would order the two.  One PPCG inner step, and a Chebyshev cap one past a checked iteration, in each on-chip
form: the sweeps' launches, and the same bits in every field."""
import numpy as np
import pytest

from helpers import small_deck

pytestmark = pytest.mark.gpu

SIZES = [(9, 9), (97, 131), (600, 433), (1003, 1201)]


@pytest.mark.parametrize("precond", ["none", "jac_diag"])
@pytest.mark.parametrize("size", SIZES, ids=["%dx%d" % s for s in SIZES])
def test_one_ppcg_inner_step(size, precond, monkeypatch):
    from tealeaf_ref_gb300 import native

    d = small_deck(nx=size[0], ny=size[1], solver="ppcg", precond=precond, ppcg_inner_steps=1, ch_cg_presteps=6,
                   ch_cg_epslim=1e30, max_iters=14, steps=2)
    fields = ["u", "w", "r", "p", "sd", "rtemp", "utemp"] + (["z"] if precond == "jac_diag" else [])
    runs = []
    for form in ("0", "1"):
        monkeypatch.setenv("TL_POLY_PERSISTENT", form)
        with native.Chunk.from_deck(d) as c:
            infos = [c.tea_leaf(d) for _ in range(2)]
            runs.append((infos, {f: c.download(f) for f in fields}))
    (i0, f0), (i1, f1) = runs
    assert sum(i.ppcg_inner_iters for i in i0) > 0
    for a, b in zip(i0, i1):
        assert (a.n_exit, a.error, a.ppcg_inner_iters, a.kernel_launches) == \
               (b.n_exit, b.error, b.ppcg_inner_iters, b.kernel_launches)
    for f in fields:
        assert np.array_equal(f0[f], f1[f]), f


@pytest.mark.parametrize("precond", ["none", "jac_diag"])
@pytest.mark.parametrize("size", SIZES[1:], ids=["%dx%d" % s for s in SIZES[1:]])
def test_one_chebyshev_iteration_after_a_check(size, precond, monkeypatch):
    from tealeaf_ref_gb300 import native

    def solve(form, cap):
        monkeypatch.setenv("TL_POLY_PERSISTENT", form)
        d = small_deck(nx=size[0], ny=size[1], solver="chebyshev", precond=precond, ch_cg_presteps=6,
                       ch_cg_epslim=1e30, max_iters=cap, steps=1)
        with native.Chunk.from_deck(d) as c:
            i = c.tea_leaf(d)
            return i, {f: c.download(f) for f in ("u", "w", "r", "p")}

    est = solve("0", 40)[0].est_itc  # from the eigenvalues, so the cap does not change it
    checked = max(est + 9, 40) // 10 * 10
    i0, f0 = solve("0", checked + 1)
    i1, f1 = solve("1", checked + 1)
    before = solve("1", checked)[0]
    assert i0.reported_iterations == checked + 1 and before.reported_iterations == checked, "converged before the cap"
    assert i1.kernel_launches < i0.kernel_launches, "the on-chip steps did not run"
    # the sweep and the copy of u back from its second field, or the kernels of a preconditioned iteration:
    # on chip it would be one launch
    assert i1.kernel_launches - before.kernel_launches >= 2
    assert (i0.n_exit, i0.error, i0.cheby_calc_steps) == (i1.n_exit, i1.error, i1.cheby_calc_steps)
    for f in f0:
        assert np.array_equal(f0[f], f1[f]), f
