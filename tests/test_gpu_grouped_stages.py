"""Batches whose labels go to the host group by group: that the groups run at all (more
launches than the same batch in one), that every stage keeps its own device time, and
that batches in flight on several slots of a server, each with its groups, give the
labels of one group."""
import time

import numpy as np
import pytest

from voxelfragmentml_gb300 import vessel as Vs

pytestmark = pytest.mark.gpu

DIMS = [(150, 149, 160), (160, 151, 161), (40, 41, 42), (170, 165, 163), (150, 160, 166), (130, 128, 131), (180, 180, 192)]


def _specs(vf, pinned, tag=0):
    specs = []
    for i, d in enumerate(DIMS):
        v, f = Vs.vessel_mesh(40 + i, 30, i)
        p = vf.Params.default(algorithm=vf.FLOOD, distance=i % 3, num_seeds=5 + i, seed=i + 1, seed_location=vf.BOTH,
                              noise_amplitude=2.0, noise_period=16)
        specs.append(vf.JobSpec(v, f, p, dims=d, aabb=Vs.mesh_aabb(v), ncounts=256, pinned=pinned, tag=tag + i))
    return specs


def _check(one, many):
    """Stage times and launches of a batch in one group and in several."""
    assert many[1] > one[1]
    for k in ("fracture", "perturb", "erode_boundaries", "counts"):
        assert many[0][k] >= 0.5 * one[0][k] > 0, (k, one[0], many[0])


def _last(ctx):
    return ctx.stage_ms(), ctx.last_stats()["launches"]


def test_stage_times_by_groups(vf, ctx):
    one, many = _specs(vf, False), _specs(vf, True)
    for _ in range(2):
        vf.batch_run(one, ctx)
        a = _last(ctx)
        vf.batch_run(many, ctx)
        b = _last(ctx)
    _check(a, b)
    rb = vf.ResidentBatch(many, ctx)
    for _ in range(3):
        rb.execute(download=True)
        assert rb.graph
        ms, launches = _last(ctx)
        assert launches > a[1]  # a replayed graph: all stages after the flood in one entry
        assert ms["perturb"] >= 0.5 * sum(a[0][k] for k in ("perturb", "erode_boundaries", "counts"))
    rb.execute(download=False)  # nothing to download: one group
    assert _last(ctx)[1] < b[1]


def test_groups_in_flight(vf, ctx):
    one = _specs(vf, False)
    vf.batch_run(one, ctx)
    batches = [_specs(vf, True, tag=7 * k) for k in range(5)]
    srv = vf.Server(ctx, max_inflight=3, max_batch=7)
    try:
        for b in batches:
            for s in b:
                srv.submit(s)
        got = []
        deadline = time.time() + 120
        while len(got) < 35 and time.time() < deadline:
            got += srv.poll(64, wait_ms=100)
        assert sorted(r.user_tag for r in got) == list(range(35)) and all(r.status == 0 for r in got)
    finally:
        srv.close()
    for b in batches:
        for s, w in zip(b, one):
            assert np.array_equal(s.labels, w.labels) and np.array_equal(s.counts, w.counts)
