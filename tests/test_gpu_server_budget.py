"""Server admission where the jobs of a micro-batch need more device memory together
than one by one: the floods of a batch share the state width of its widest job (8
words a row up to 64 seeds, 16 above 1024).  Every admitted job must run."""
import time

import numpy as np
import pytest

from voxelfragmentml_gb300 import vessel as Vs

pytestmark = pytest.mark.gpu


def _spec(vf, i, extra=0):
    v, f = Vs.vessel_mesh(40, 30, i % 3)
    p = vf.Params.default(num_seeds=100 if extra else 8, num_extra_seeds=extra, seed=i + 1)
    return vf.JobSpec(v, f, p, dims=(200, 197, 208), aabb=Vs.mesh_aabb(v), ncounts=256, tag=i, want_labels=False)


def _specs(vf):
    return [_spec(vf, i) for i in range(24)] + [_spec(vf, 24, extra=1100)]


def test_admission_of_mixed_state_widths(vf, ctx):
    want, specs = _specs(vf), _specs(vf)
    vf.batch_run(want, ctx)
    # what the 25 jobs need one by one, and 64 MB for the rounding of some 40 arenas to
    # 1 MB each; at the widest job's width they need 24 * 325 k rows * 32 bytes more
    jobs = [s.job() for s in specs]
    budget = sum(vf.lib().vf_job_footprint(vf.C.byref(j)) for j in jobs) + (64 << 20)
    c = vf.Context(0, hbm_budget=budget)
    srv = vf.Server(c, hbm_budget=budget, max_inflight=1, max_batch=64)
    try:
        first = _spec(vf, 25)  # keeps the slot busy while the others queue up
        for s in [first] + specs:
            srv.submit(s)
        got = []
        deadline = time.time() + 120
        while len(got) < len(specs) + 1 and time.time() < deadline:
            got += srv.poll(64, wait_ms=100)
        assert sorted(r.user_tag for r in got) == list(range(26))
        assert [r.status for r in got] == [0] * 26
        for a, b in zip(specs, want):
            assert np.array_equal(a.counts, b.counts)
    finally:
        srv.close()
        c.close()
