"""Batches whose labels go to the host group by group (csrc/vf_runtime.cu,
plan_groups): pinned labels of 32 MB or more in all, ragged rows, jobs without
labels, every stage after the flood, resident runs.  Labels and counts must equal
those of the same jobs with pageable labels (one group), and one job the oracle's."""
import numpy as np
import pytest

import oracle as O
from voxelfragmentml_gb300 import vessel as Vs

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _oracle(oracle_lib):
    return oracle_lib


DIMS = [(150, 149, 160), (160, 151, 161), (40, 41, 42), (170, 165, 163), (150, 160, 166), (130, 128, 131), (180, 180, 192)]


def _specs(vf, pinned, prefix=False):
    specs = []
    for i, d in enumerate(DIMS):
        v, f = Vs.vessel_mesh(40 + i, 30, i)
        p = vf.Params.default(algorithm=vf.NAIVE if i == 1 else vf.FLOOD, distance=i % 3, num_seeds=5 + i, seed=i + 1,
                              seed_location=vf.BOTH, noise_amplitude=2.0 if i % 2 else 0.0, noise_period=16,
                              boundary_size=3 if i == 4 else 1)
        if i in (0, 5):
            p.erode, p.erosion_type, p.erosion_size, p.erosion_iterations = 1, vf.SQUARE, 3, 1 + i % 2
        if prefix and i == 3:
            p.num_extra_seeds = 9
        specs.append(vf.JobSpec(v, f, p, dims=d, aabb=Vs.mesh_aabb(v), ncounts=256 + i, pinned=pinned,
                                want_labels=i != 2))
    return specs


def _same(a, b):
    for x, y in zip(a, b):
        assert (x.labels is None) == (y.labels is None)
        assert x.labels is None or np.array_equal(x.labels, y.labels)
        assert np.array_equal(x.counts, y.counts)


@pytest.mark.parametrize("prefix", [False, True])
def test_groups(vf, ctx, prefix):
    one, many = _specs(vf, False, prefix), _specs(vf, True, prefix)
    for r in vf.batch_run(one, ctx) + vf.batch_run(many, ctx):
        assert r.status == 0
    _same(one, many)
    s = many[5]
    q = O.Params()
    for name, _ in O.Params._fields_:
        setattr(q, name, getattr(s.params, name))
    want = O.run_job(s.verts, s.faces, s.dims, s.aabb[0], s.aabb[1], q, ncounts=len(s.counts))
    assert np.array_equal(s.labels, want[0]) and np.array_equal(s.counts, want[1])


def test_resident_groups(vf, ctx):
    one, many = _specs(vf, False), _specs(vf, True)
    vf.batch_run(one, ctx)
    b = vf.ResidentBatch(many, ctx)
    for download in (True, False, True):
        for s in many:
            if s.labels is not None and download:
                s.labels[...] = 7
            s.counts[...] = 0
        for r in b.execute(download=download):
            assert r.status == 0
        if download:
            _same(one, many)
