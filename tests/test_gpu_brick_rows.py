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


def _labels(shape, seed):
    rng = np.random.default_rng(seed)
    lab = rng.integers(0, 5, [(s + 6) // 7 for s in shape]).astype(np.uint16)
    for a in range(3):
        lab = np.repeat(lab, 7, axis=a)
    lab = np.ascontiguousarray(lab[: shape[0], : shape[1], : shape[2]])
    lab[rng.random(shape) < 0.02] = 0
    return lab


@pytest.mark.parametrize("period", [1, 3, 5, 6, 7, 15, 16, 17, 40, 1000])
@pytest.mark.parametrize("shape", [(2, 3, 2), (33, 35, 66), (16, 16, 32), (40, 17, 100)])
def test_perturb(vf, ctx, shape, period):
    lab = _labels(shape, period)
    for amp in (0.7, 5.0, 64.0):
        g = vf.RegularGrid(shape, None, None, ctx)
        g.upload(lab)
        g.perturb(amp, period, 9)
        assert np.array_equal(g.data(), O.perturb(lab, amp, period, 9))
        g.close()


@pytest.mark.parametrize("shape", [(2, 3, 2), (16, 16, 32), (33, 35, 66), (9, 40, 130)])
@pytest.mark.parametrize("labels", [3, 255, 256, 300])
def test_counts(vf, ctx, shape, labels):
    rng = np.random.default_rng(labels)
    lab = _labels(shape, 1)
    noisy = rng.random(shape) < 0.3
    lab[noisy] = rng.integers(0, labels + 1, int(noisy.sum()))
    lab |= (rng.random(shape) < 0.3).astype(np.uint16) << 15
    g = vf.RegularGrid(shape, None, None, ctx)
    g.upload(lab)
    want = np.bincount((lab & 0x7FFF)[(lab > 1)].ravel(), minlength=512)[:512]
    counts, occupied = g.countValues(512)
    assert np.array_equal(counts[2:], want[2:]) and occupied == (lab > 1).sum()
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
