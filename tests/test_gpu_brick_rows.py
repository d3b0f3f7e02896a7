"""Brick kernels whose rules changed with the row length, the noise period and
the planes a flood starts from: rows of 1 to 512 units through the fill, the
perturbation around the lattice table's size, counts of runs and mixed rows, a
job's flood.  Bit for bit against the oracle."""
import numpy as np
import pytest

import oracle as O
from voxelfragmentml_gb300 import vessel as Vs

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _oracle(oracle_lib):
    return oracle_lib


@pytest.mark.parametrize("dims", [(2, 2, 2), (17, 16, 8), (16, 33, 9), (31, 18, 72), (20, 20, 257), (5, 6, 2049),
                                  (3, 2, 4096)])
def test_fill(vf, ctx, dims):
    v, f = Vs.vessel_mesh(24, 18, 3)
    mn, mx = Vs.mesh_aabb(v)
    g = vf.RegularGrid(dims, mn, mx, ctx)
    g.fill(v, f)
    assert np.array_equal(g.data(), O.voxelize(v, f, dims, mn, mx))
    g.detectBoundaries(1)  # reads the second buffer's bricks as zeros around the live ones
    g.close()
