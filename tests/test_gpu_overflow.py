"""Sums beyond the range of FP64 in the on-chip CG loops: an infinite p.w with a finite r.r makes alpha
zero and the loop runs on, as in the sweeps; an infinite r.r breaks both down."""
import numpy as np
import pytest

from helpers import small_deck

pytestmark = pytest.mark.gpu


def run(d, form, monkeypatch):
    from tealeaf_ref_gb300 import native

    monkeypatch.setenv("TL_CG_PERSISTENT", form)
    with native.Chunk.from_deck(d) as c:
        try:
            i = c.tea_leaf(d)
        except native.TeaLeafError as e:
            return e.code, None, None
        return 0, i, c.download("u")


@pytest.mark.parametrize("size", [(20, 20), (64, 64), (512, 512), (1003, 1001)], ids=lambda s: "%dx%d" % s)
@pytest.mark.parametrize("rr", [1.0e308, float("inf")], ids=["pw", "rr"])
def test_overflowing_sums(size, rr, monkeypatch):
    d = small_deck(nx=size[0], ny=size[1], steps=1, max_iters=4)
    _, i, _ = run(d, "0", monkeypatch)
    root = rr ** 0.5 if rr < float("inf") else 1.0e156
    for s in d.states:
        s.energy *= root / i.initial_residual
    (c0, i0, u0), (c1, i1, u1) = run(d, "0", monkeypatch), run(d, "1", monkeypatch)
    assert c0 == c1
    if c0 == 0:
        assert i1.kernel_launches < i0.kernel_launches, "the on-chip loop did not run"
        assert (i0.n_exit, i0.cg_calc_steps) == (i1.n_exit, i1.cg_calc_steps)
        assert abs(i1.error - i0.error) <= 1e-12 * i0.error
        assert np.array_equal(u0, u1)  # alpha is zero throughout
