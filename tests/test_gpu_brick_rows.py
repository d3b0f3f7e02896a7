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


@pytest.mark.parametrize("dims", [(2, 2, 2), (16, 31, 33), (40, 38, 64), (7, 50, 129)])
@pytest.mark.parametrize("dfunc", [0, 1, 2])
def test_job(vf, ctx, dims, dfunc):
    # the flood of a job starts from the voxelizer's bit planes
    v, f = Vs.vessel_mesh(20, 15, 2)
    mn, mx = Vs.mesh_aabb(v)
    p = vf.Params.default(distance=dfunc, num_seeds=1 if dims[0] < 4 else 9, seed=5, seed_location=vf.BOTH)
    spec = vf.JobSpec(v, f, p, dims=dims, aabb=(mn, mx), ncounts=256)
    r = vf.batch_run([spec], ctx)[0]
    q = O.Params()
    for name, _ in O.Params._fields_:
        setattr(q, name, getattr(p, name))
    want = O.run_job(v, f, dims, mn, mx, q, ncounts=256)
    assert r.status == 0
    assert np.array_equal(spec.labels, want[0]) and np.array_equal(spec.counts, want[1][:256])
