"""vf_autotune decides what changes a launch, and leaves the rest as the caller set it:
the flood has no sweeps, and no third CTA per SM."""
import pytest

from voxelfragmentml_gb300 import vessel as Vs

pytestmark = pytest.mark.gpu


def _spec(vf, i):
    v, f = Vs.vessel_mesh(24, 18, i)
    p = vf.Params.default(num_seeds=4, seed=i + 1)
    return vf.JobSpec(v, f, p, dims=(40, 40, 44 + i), aabb=Vs.mesh_aabb(v), ncounts=256, want_labels=False)


@pytest.mark.parametrize("jobs", [1, 4])
def test_autotune_leaves_what_nothing_reads(vf, ctx, jobs):
    saved = ctx.tuning()
    try:
        ctx.set_tuning(flood_sweeps=5, flood_ctas=2)
        chosen = ctx.autotune([_spec(vf, i) for i in range(jobs)])
        assert chosen["flood_sweeps"] == 5
        assert chosen["flood_ctas"] == 0
        assert chosen["parity_grid"] in (4, 8, 16, 32) and chosen["shell_grid"] in (6, 12, 24)
        assert ctx.tuning() == chosen
    finally:
        ctx.set_tuning(**saved)
