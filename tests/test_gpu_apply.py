"""The drop-in kernels w = A p (with p.w) and r = u0 - A u on meshes large enough for their staged
form, against the same operator in numpy from the downloaded face coefficients: ragged strips, an odd
width, a mesh narrower than a strip.

Each value is a sum of five products: the two orders of evaluation and the scaled faces' own rounding
(one more factor) leave at most 8 units of 2^-53 of the terms' magnitudes between them; the sum p.w of
n terms n units of the sum of their magnitudes."""
import numpy as np
import pytest

from helpers import small_deck

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("size", [(2048, 1025), (2049, 1024), (4099, 513), (255, 8300)], ids=lambda s: "%dx%d" % s)
def test_staged_operator_matches_the_plain_one(size):
    from tealeaf_ref_gb300 import native

    nx, ny = size
    rng = np.random.default_rng(5)
    d = small_deck(nx=nx, ny=ny, n_rect=6, n_circ=2)
    with native.Chunk.from_deck(d) as c:
        c.common_init(0.004)
        kx, ky, di = (c.download(f) for f in ("kx", "ky", "di"))
        v = rng.standard_normal((ny, nx))
        c.upload("p", v)
        c.upload("u", v)
        pw = c.cg_calc_w()
        c.calc_residual()
        w, r, u0 = c.download("w"), c.download("r"), c.download("u0")
    # the plain product in numpy, with the scaled faces, to the rounding of its few terms
    rx, ry = 0.004 / d.dx ** 2, 0.004 / d.dy ** 2
    cx, cy = rx * kx, ry * ky
    want = di * v
    scale = np.abs(want)
    for sl, nb, co in (((slice(1, None), slice(None)), (slice(0, -1), slice(None)), cy),
                       ((slice(None), slice(1, None)), (slice(None), slice(0, -1)), cx)):
        want[sl] -= co[sl] * v[nb]
        want[nb] -= co[sl] * v[sl]
        scale[sl] += np.abs(co[sl] * v[nb])
        scale[nb] += np.abs(co[sl] * v[sl])
    assert np.all(np.abs(w - want) <= 8 * 2.0 ** -53 * scale)
    assert np.all(np.abs(r - (u0 - want)) <= 9 * 2.0 ** -53 * (scale + np.abs(u0)))
    assert abs(pw - float(np.sum(v * want))) <= 2.0 ** -53 * nx * ny * float(np.sum(np.abs(v) * scale))
