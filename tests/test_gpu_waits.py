"""The bounded waits of the on-chip loops.  A wait that runs out makes the solve return TL_ERR_TIMEOUT,
and the context then solves normally; also when one tile alone fails in the last iteration and every
other tile, the one that stores the loop's state among them, ends its loop as usual."""
import pytest

from helpers import small_deck

pytestmark = pytest.mark.gpu

TL_ERR_TIMEOUT = -5

# k_persistent_cg, k_persistent_cg_wide; k_persistent_mix with groups of two and of four rows
CG_FORMS = [("fp64", 64, 64), ("fp64", 1003, 1001), ("mixed", 200, 160), ("mixed", 1000, 1000)]
CG_IDS = ["%s-%dx%d" % f for f in CG_FORMS]


def check(d, opts, fault, monkeypatch):
    from tealeaf_ref_gb300 import native

    with native.Chunk.from_deck(d) as c:
        want = c.tea_leaf(opts, d.initial_timestep)
        c.generate(d)
        c.reset_eigen()
        monkeypatch.setenv("TL_CG_BARRIER_EXTRA", fault)
        with pytest.raises(native.TeaLeafError) as e:
            c.tea_leaf(opts, d.initial_timestep)
        assert e.value.code == TL_ERR_TIMEOUT
        monkeypatch.delenv("TL_CG_BARRIER_EXTRA")
        c.generate(d)
        c.reset_eigen()
        got = c.tea_leaf(opts, d.initial_timestep)
        assert (got.n_exit, got.error) == (want.n_exit, want.error)


def cg_opts(precision, nx, ny, iters):
    from tealeaf_ref_gb300 import native

    d = small_deck(nx=nx, ny=ny, steps=1, max_iters=iters)
    o = native.opts_from_deck(d, precision, max_inner_iters=iters) if precision == "mixed" else native.opts_from_deck(d)
    return d, o


@pytest.mark.parametrize("form", CG_FORMS, ids=CG_IDS)
def test_a_sum_that_never_completes(form, monkeypatch):
    check(*cg_opts(*form, 20), "1", monkeypatch)


@pytest.mark.parametrize("form", CG_FORMS, ids=CG_IDS)
def test_one_tile_that_gives_up_in_the_last_iteration(form, monkeypatch):
    check(*cg_opts(*form, 1), "3", monkeypatch)


@pytest.mark.parametrize("solver", ["ppcg", "chebyshev"])
def test_a_rim_that_never_comes_on_larger_tiles(solver, monkeypatch):
    from tealeaf_ref_gb300 import native

    d = small_deck(nx=1003, ny=1201, solver=solver, ppcg_inner_steps=6, ch_cg_presteps=10, ch_cg_epslim=1e30,
                   max_iters=40, steps=1)
    check(d, native.opts_from_deck(d), "2", monkeypatch)
