"""The second label buffer between stages that swap buffers: their tiles read the bricks
around a live one from it, also the ones that are not live, which the fill must have
cleared there (k_combine).  A small model filled where a large one was fractured, through
perturbation, two erosions and the removal of isolated voxels, against the oracle."""
import numpy as np
import pytest

import oracle as O
from voxelfragmentml_gb300 import vessel as Vs

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _oracle(oracle_lib):
    return oracle_lib


@pytest.mark.parametrize("dims", [(17, 33, 40), (31, 18, 72), (20, 20, 257), (48, 35, 65)])
def test_refilled_grid(vf, ctx, dims):
    v, f = Vs.vessel_mesh(24, 18, 3)
    mn, mx = Vs.mesh_aabb(v)
    mn, mx = np.array(mn, np.float32), np.array(mx, np.float32)
    mid = (mn + mx) / 2
    g = vf.RegularGrid(dims, mn, mx, ctx)
    for k, shrink in enumerate((1.0, 0.45, 1.0, 0.3)):
        # not in the middle: bricks that were live stay empty beside it
        w = np.ascontiguousarray(((v - mid) * shrink + mid - (1 - shrink) * 0.4 * (mx - mn)).astype(np.float32))
        p = vf.Params.default(distance=k % 3, num_seeds=4 + k, seed=k + 5, seed_location=vf.BOTH, noise_amplitude=3.0,
                              noise_period=6, erode=1, erosion_type=vf.SQUARE, erosion_size=3, erosion_iterations=2)
        g.fill(w, f)
        vf.fracture_model(g, p)
        q = O.Params()
        for name, _ in O.Params._fields_:
            setattr(q, name, getattr(p, name))
        want = O.run_job(w, f, dims, mn, mx, q, ncounts=256)[0]
        assert want.any() and np.array_equal(g.data(), want)
    g.close()
