"""The tilings of the on-chip CG kernel, and the exchange of the tiles' rims, by the kernel's own index
arithmetic on the CPU: every tile is owned cell by cell, every word a thread polls in its tile's halo box
is written by exactly one owner of the neighbouring tile and holds the cell beside it, and every box
lies in the allocation.  So every wait ends and no access leaves its buffer.

Meshes of 400 to 12000 cells ran in one thread-block cluster before, whose CTAs exchanged through each
other's shared memory; that form raised a fault under a profiler.  No kernel uses a cluster now."""
import ctypes
import glob
import os
import re

import pytest

from tealeaf_ref_gb300 import build

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CTAS = 152       # SMs of a GB300
OWNERS = 480     # threads of a CTA that own cells
HALO_CELLS = 2   # halo cells a thread fetches at most
INBOX = 160      # words of an inbox
VARIANTS = [1, 2, 4, 6, 8, 11]


class Plan(ctypes.Structure):
    _fields_ = [(n, ctypes.c_int) for n in ("gx", "gy", "tw", "th", "ry", "variant", "rows")]


@pytest.fixture(scope="module")
def lib():
    return ctypes.CDLL(build.build())


def plan_of(lib, nx, ny):
    p = Plan()
    fn = lib._ZN2tl12persist_planEiiiPNS_11PersistPlanE
    fn.restype = ctypes.c_bool
    return p if fn(nx, ny, CTAS, ctypes.byref(p)) else None


def box_bytes(lib, p):
    fn = lib._ZN2tl17persist_box_bytesERKNS_11PersistPlanE
    fn.restype = ctypes.c_size_t
    return fn(ctypes.byref(p))


def test_no_kernel_of_the_library_uses_a_cluster():
    for f in glob.glob(os.path.join(ROOT, "tealeaf_ref_gb300", "csrc", "*.cu*")):
        src = open(f).read()
        assert not re.search(r"barrier\.cluster|\bmapa\b|ClusterDimension|__cluster_dims__|cluster_group", src), f


SIZES = ([(n, n) for n in (2, 10, 15, 19, 20, 21, 22, 33, 48, 61, 64, 96, 97, 105, 110, 127, 256, 512, 700)]
         + [(1, 2), (1, 400), (401, 1), (1, 900), (900, 1), (3, 4000), (4000, 3), (1, 20000), (20000, 3), (37, 23),
            (301, 40), (105, 104), (301, 499), (777, 813)])


@pytest.mark.parametrize("size", SIZES, ids=["%dx%d" % s for s in SIZES])
def test_tiles_and_rims(lib, size):
    nx, ny = size
    p = plan_of(lib, nx, ny)
    assert p is not None
    ctas, hbox, P = p.gx * p.gy, 2 * (p.th + p.tw), p.tw + 2
    assert 1 <= ctas <= CTAS
    assert (p.gx - 1) * p.tw < nx <= p.gx * p.tw and (p.gy - 1) * p.th < ny <= p.gy * p.th
    assert p.ry * p.tw <= OWNERS and hbox <= HALO_CELLS * OWNERS
    assert -(-p.th // p.ry) <= VARIANTS[p.variant]
    assert 4 * 8 * (p.th + 2) * P <= 225 * 1024
    assert 16 * ctas * (2 * INBOX + hbox) <= box_bytes(lib, p)  # the two inboxes of a CTA, then the halo boxes

    sent = {}  # word of the halo boxes -> the cell its writer puts there
    owned = 0
    for b in range(ctas):
        bx, by = b % p.gx, b // p.gx
        j0, k0 = bx * p.tw, by * p.th
        tw, th = min(p.tw, nx - j0), min(p.th, ny - k0)
        for to in range(p.ry * p.tw):
            tx, ty = to % p.tw, to // p.tw
            mine = (th - 1 - ty) // p.ry + 1 if tx < tw and ty < p.ry and ty < th else 0
            owned += mine
            i_first = 0 if ty == 0 else -1
            i_last = mine - 1 if mine > 0 and (th - 1 - ty) % p.ry == 0 else -1
            to_l = (b - 1) * hbox + p.th + ty if tx == 0 and j0 > 0 else -1
            to_r = (b + 1) * hbox + ty if tx == tw - 1 and j0 + tw < nx else -1
            rim_b = i_first if k0 > 0 else -1
            rim_t = i_last if k0 + th < ny else -1
            for i in range(mine):
                cell = (j0 + tx, k0 + ty + i * p.ry)
                words = []
                if to_l >= 0:
                    words.append(to_l + i * p.ry)
                if to_r >= 0:
                    words.append(to_r + i * p.ry)
                if i == rim_b:
                    words.append((b - p.gx) * hbox + 2 * p.th + p.tw + tx)
                if i == rim_t:
                    words.append((b + p.gx) * hbox + 2 * p.th + tx)
                for w in words:
                    assert 0 <= w < ctas * hbox and w not in sent
                    sent[w] = cell
    assert owned == nx * ny
    polled = {}
    for b in range(ctas):
        bx, by = b % p.gx, b // p.gx
        j0, k0 = bx * p.tw, by * p.th
        tw, th = min(p.tw, nx - j0), min(p.th, ny - k0)
        for h in range(hbox):
            x, y, there = -1, h, j0 > 0 and h < th
            if h >= p.th:
                x, y = tw, h - p.th
                there = j0 + tw < nx and y < th
            if h >= 2 * p.th:
                x, y = h - 2 * p.th, -1
                there = k0 > 0 and x < tw
            if h >= 2 * p.th + p.tw:
                x, y = h - 2 * p.th - p.tw, th
                there = k0 + th < ny and x < tw
            if there:
                assert 0 <= (y + 1) * P + x + 1 < (p.th + 2) * P
                polled[b * hbox + h] = (j0 + x, k0 + y)
    assert polled == sent
