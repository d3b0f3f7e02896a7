"""Floods of large flat grids (csrc/vf_flood.cu, wave_order): words along the longest
axis from 4 M rows on where z has few voxels.  Either axis, sub-seeds, seeds on empty
voxels, whole jobs beside ones with words along z, against the oracle; and the device
memory they take."""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _oracle(oracle_lib):
    return oracle_lib


@pytest.mark.parametrize("shape,frac,prefixes,dfunc", [
    ((2048, 1100, 2), 0.9, 0, 1), ((1100, 2049, 3), 0.7, 0, 2), ((2047, 1101, 4), 0.8, 3, 2), ((1031, 2100, 2), 1.0, 2, 1),
    ((1100, 2048, 9), 0.8, 0, 1)])  # the last: words along z
def test_flat_floods(vf, ctx, shape, frac, prefixes, dfunc):
    rng = np.random.default_rng(sum(shape))
    occ = (rng.random(shape) < frac).astype(np.uint16)
    n = 70  # two plane counts
    at = np.stack([rng.integers(0, s, n) for s in shape], 1)
    label = np.arange(n) % 60 + 2
    if prefixes:
        label = label % 9 + 2 | (rng.integers(0, prefixes, n) << 8)
    seeds = np.concatenate([at, label[:, None]], axis=1).astype(np.uint32)
    want = O.flood(occ, seeds, dfunc)[0]
    g = vf.RegularGrid(shape, None, None, ctx)
    g.upload(occ)
    fr = vf.FloodFracturer()
    fr.setDistanceFunction(dfunc)
    fr.build(g, seeds)
    got = g.data()
    g.close()
    assert np.array_equal(got, want)


BOX_V = np.array([[x, y, z] for x in (0, 1) for y in (0, 1) for z in (0, 1)], np.float32)
BOX_F = np.array([[0, 1, 3], [0, 3, 2], [4, 6, 7], [4, 7, 5], [0, 4, 5], [0, 5, 1], [2, 3, 7], [2, 7, 6],
                  [0, 2, 6], [0, 6, 4], [1, 5, 7], [1, 7, 3]], np.uint32)


def test_flat_jobs_in_a_batch(vf, ctx):
    specs = []
    for i, dims in enumerate([(60, 50, 40), (2048, 1100, 2), (33, 90, 64), (1100, 2049, 3), (200, 200, 8)]):
        p = vf.Params.default(distance=i % 3, num_seeds=5 + i, seed=i + 1, seed_location=vf.BOTH,
                              num_extra_seeds=9 if i == 3 else 0)
        specs.append(vf.JobSpec(BOX_V, BOX_F, p, dims=dims, aabb=((-0.1, 0.0, 0.0), (1.3, 1.0, 1.0)), ncounts=256,
                                pinned=bool(i % 2)))
    for r, s in zip(vf.batch_run(specs, ctx), specs):
        assert r.status == 0
        q = O.Params()
        for name, _ in O.Params._fields_:
            setattr(q, name, getattr(s.params, name))
        lab, cnt = O.run_job(s.verts, s.faces, s.dims, s.aabb[0], s.aabb[1], q, ncounts=256)[:2]
        assert np.array_equal(s.labels, lab) and np.array_equal(s.counts, cnt)


def test_flat_flood_memory(vf):
    """4096 x 4096 x 2 voxels: labels twice 0.54 GB and bit planes 0.13 GB; the flood's state
    with words along z would add 1.65 GB."""
    p = vf.Params.default(num_seeds=8)
    spec = vf.JobSpec(BOX_V, BOX_F, p, dims=(4096, 4096, 2), aabb=((0.0, 0.0, 0.0), (1.0, 1.0, 1.0)), ncounts=256,
                      want_labels=False)
    j = spec.job()
    assert vf.lib().vf_job_footprint(vf.C.byref(j)) < 1 << 30
