"""The face coefficients and Di of the set-up against numpy, at sizes where a thread marches up 1, 4, 9
and 32 rows, with ragged last strips and marches.  Both sides do the same IEEE operations in the same
order: the same bits."""
import numpy as np
import pytest

from helpers import small_deck

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("coefficient", [1, 2])
@pytest.mark.parametrize("reflective", [False, True])
@pytest.mark.parametrize("size", [(10, 10), (1, 5000), (257, 3000), (2000, 1500), (4001, 3001)],
                         ids=lambda s: "%dx%d" % s)
def test_faces_have_the_bits_of_the_formula(size, reflective, coefficient):
    from tealeaf_ref_gb300 import native

    nx, ny = size
    d = small_deck(nx=nx, ny=ny, steps=1, coefficient=coefficient, reflective=reflective, max_iters=1)
    dt = d.initial_timestep
    with native.Chunk.from_deck(d) as c:
        rho = np.random.default_rng(3).uniform(0.1, 100.0, (ny, nx))
        c.upload_state(rho, np.ones((ny, nx)))
        c.common_init(dt)
        kx, ky, di = (c.download(f) for f in ("kx", "ky", "di"))
    w = np.pad(1.0 / rho if coefficient == 2 else rho, 1, mode="edge")

    def face(a, b):
        return (a + b) / ((2.0 * a) * b)

    x = face(w[1:-1, :-1], w[1:-1, 1:])  # faces 1 .. nx + 1
    y = face(w[:-1, 1:-1], w[1:, 1:-1])
    if not reflective:
        x[:, 0] = x[:, -1] = 0.0
        y[0] = y[-1] = 0.0
    dx, dy = (d.xmax - d.xmin) / nx, (d.ymax - d.ymin) / ny
    rx, ry = dt / (dx * dx), dt / (dy * dy)
    assert np.array_equal(kx, x[:, :-1])
    assert np.array_equal(ky, y[:-1])
    assert np.array_equal(di, (1.0 + ry * (y[1:] + y[:-1])) + rx * (x[:, 1:] + x[:, :-1]))
