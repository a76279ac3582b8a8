"""Detector cells coarser than a voxel, and rows that span more slices than a
window: the projector's forms for rays that are not narrow, with the bits of the
plain loops."""
import numpy as np
import pytest

from conftest import geo
from test_gpu_aligned_copies import program, run  # noqa: F401 (a fixture)
from test_gpu_kernels import GEOS  # the projector parity geometries

pytestmark = pytest.mark.gpu

# (da, db): footprints of up to 2, 3 and more voxels in-plane and slices high
CELLS = [(0.9, 1.6), (1.6, 1.6), (2.3, 2.3), (2.6, 3.1), (4.5, 4.4), (0.7, 2.9), (2.9, 0.7),
         (0.9, 1.45), (6.1, 0.3)]


def test_wide_footprints_have_the_plain_loops_bits(program):
    cases = []
    for da, db in CELLS:
        for nx, ny, nz, na, nb in ((44, 40, 41, 30, 37), (33, 65, 6, 7, 70)):
            g = geo(nx=nx, ny=ny, nz=nz, na=na, nb=nb, SO=90.0, SD=135.0, da=da, db=db, ai=0.37, bi=-0.61)
            cases += [(g, nz + nz % 2, angle) for angle in (0.3, 0.7853982, 1.5, 3.9)]
    run(program, cases)


def test_the_forms_that_geometries_take(program):
    """The parity geometries take the staged forms at the volume's inside and edge; with
    the cells above, and narrow rays whose in-plane footprint is three voxels in some
    slabs only, every form is taken."""
    parity = run(program, [(g, g["nz"] + g["nz"] % 2, angle) for g in GEOS
                           for angle in (0.3, 0.7853, 1.5707964, 3.9)])
    assert all(n > 0 for n in np.sum(parity, axis=0)[:2]), np.sum(parity, axis=0)
    coarse = run(program, [(geo(nx=44, ny=40, nz=41, na=30, nb=37, SO=90.0, SD=135.0, da=da, db=db),
                            42, 0.6) for da, db in CELLS + [(1.45, 0.8), (3.5, 0.8)]])
    assert all(n > 0 for n in np.sum(coarse, axis=0)), np.sum(coarse, axis=0)


def test_a_source_inside_the_volume(program):
    """Rays run both ways from the source's plane, so that no edge keeps its order."""
    g = geo(nx=60, ny=56, nz=30, na=40, nb=36, SO=20.0, SD=70.0, da=1.2, db=1.1)
    run(program, [(g, 30, angle) for angle in (0.3, 1.5, 2.4)])
