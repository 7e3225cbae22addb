"""The chunk generator's mask form against its general form, bit for bit: the same states with enough
rectangles outside the domain prepended to exceed the 64 states the masks hold.  Rectangles, circles
(some reaching past the domain, into the halo; one of zero radius on a cell centre) and points, in
an order in which each kind overwrites the others; meshes at the edges of the blocks."""
import numpy as np
import pytest

from helpers import small_deck
from tealeaf_ref_gb300 import deck as dk

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("size", [(1, 1), (7, 130), (254, 62), (255, 63), (256, 64), (511, 65), (300, 211)],
                         ids=lambda s: "%dx%d" % s)
def test_masks_match_the_loop_over_states(size):
    from tealeaf_ref_gb300 import native

    d = small_deck(nx=size[0], ny=size[1], n_rect=9, n_circ=6, seed=31, reflective=True)
    hx, hy = 10.0 / size[0], 10.0 / size[1]
    d.states += [
        dk.State(density=0.3, energy=3.0, geometry=2, xmin=0.1, ymin=9.9, radius=2.0),
        dk.State(density=0.4, energy=4.0, geometry=3, xmin=hx * (size[0] // 2), ymin=hy * (size[1] // 3)),
        dk.State(density=0.5, energy=5.0, geometry=1, xmin=4.0, xmax=6.0, ymin=3.0, ymax=9.0),
        dk.State(density=0.6, energy=6.0, geometry=2, xmin=0.5 * hx - hx / 100, ymin=0.5 * hy - hy / 100, radius=0.0),
        dk.State(density=0.7, energy=7.0, geometry=3, xmin=0.0, ymin=0.0),
    ]
    outside = [dk.State(density=9.0, energy=9.0, geometry=1, xmin=90.0, xmax=91.0, ymin=90.0, ymax=91.0)] * 64
    fields = []
    for states in (d.states, d.states[:1] + outside + d.states[1:]):
        e = d.replace(states=list(states))
        e.states = list(states)
        with native.Chunk.from_deck(e) as c:
            c.common_init(0.004)  # Kx, Ky read the density's halo
            fields.append({f: c.download(f) for f in ("density", "energy1", "kx", "ky")})
    for f in fields[0]:
        assert np.array_equal(fields[0][f], fields[1][f]), f
    if size != (1, 1):
        assert len(np.unique(fields[0]["density"])) > 3
