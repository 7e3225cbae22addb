"""The decks of test_gpu_poly_sweeps.py with the on-chip polynomial steps off: their meshes fit on chip
but for the largest, so by default the staged sweeps that those tests compare run on the largest only.
And the deck that leaves on an unchecked Chebyshev iteration, on chip against the sweeps."""
import numpy as np
import pytest

import test_gpu_poly_sweeps as sweeps
from helpers import small_deck

pytestmark = pytest.mark.gpu


@pytest.fixture
def off_chip(monkeypatch):
    monkeypatch.setenv("TL_POLY_PERSISTENT", "0")
    return monkeypatch


@pytest.mark.parametrize("name", [n for n in sweeps.DECKS if "4000" not in n])
def test_inner_sweep(name, off_chip):
    sweeps.test_inner_sweep_gives_the_same_bits(name, off_chip)


@pytest.mark.parametrize("name", [n for n in sweeps.CHEBY_DECKS if "4000" not in n])
def test_cheby_sweep(name, off_chip):
    sweeps.test_cheby_sweep_gives_the_same_bits(name, off_chip)


def test_cheby_sweep_exit_on_an_unchecked_iteration(off_chip):
    sweeps.test_cheby_sweep_exit_on_an_unchecked_iteration(off_chip)


@pytest.mark.parametrize("precond", ["none", "jac_diag"])
def test_on_chip_exit_on_an_unchecked_iteration(precond, monkeypatch):
    from tealeaf_ref_gb300 import native

    d = small_deck(nx=600, ny=433, solver="chebyshev", precond=precond, ch_cg_presteps=20, ch_cg_epslim=1e30,
                   max_iters=300, steps=1)
    with native.Chunk.from_deck(d) as c:
        r0 = c.tea_leaf(d).initial_residual
    d.eps = 1.5 / r0
    runs = []
    for form in ("0", "1"):
        monkeypatch.setenv("TL_POLY_PERSISTENT", form)
        with native.Chunk.from_deck(d) as c:
            i = c.tea_leaf(d)
            runs.append(((i.reported_iterations, i.error, i.cheby_calc_steps),
                         {f: c.download(f) for f in ("u", "w", "r", "p")}))
    (i0, f0), (i1, f1) = runs
    assert 0 < i0[2] and i0[0] < d.max_iters, i0
    assert i1 == i0
    for f in f0:
        assert np.array_equal(f0[f], f1[f]), f
