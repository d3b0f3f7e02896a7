"""Ray batches (csrc/vf_impact.cu) where their path changes: 32768 rays, cells of
8 and of 16 voxels with ragged last ones, directions of zero.  Entry voxels must
equal the oracle's."""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _oracle(oracle_lib):
    return oracle_lib


def _rays(dims, n, rng):
    o = (rng.random((n, 3)) * 3 - 1) * dims
    to = rng.random((n, 3)) * dims
    r = np.concatenate([o, to - o], 1).astype(np.float32)
    r[::7, 3 + rng.integers(0, 3)] = 0.0  # along a plane
    r[::11, 3:5] = 0.0                    # along an axis
    r[np.all(r[:, 3:] == 0, 1), 3] = 1.0
    return r


@pytest.mark.parametrize("dims,n", [((9, 17, 33), 4095), ((9, 17, 33), 32767), ((9, 17, 33), 32768), ((2, 2, 2), 33000),
                                    ((70, 64, 95), 40001), ((12, 14, 600), 33000), ((1000, 300, 520), 33000)])
def test_entry_voxels(vf, ctx, dims, n):
    rng = np.random.default_rng(n)
    lab = np.zeros(dims, np.uint16)
    for p in rng.integers(0, dims, (40, 3)):
        lab[tuple(p)] = 1 + p[0]
    lab[dims[0] // 2:, dims[1] // 2:, -1] = 3
    mn, mx = np.zeros(3, np.float32), np.array(dims, np.float32)
    g = vf.RegularGrid(dims, mn, mx, ctx)
    g.upload(lab)
    rays = _rays(np.array(dims), n, rng)
    assert np.array_equal(g.rayEntryVoxels(rays), O.ray_entry_batch(lab, mn, mx, rays))
    g.close()


@pytest.mark.parametrize("n", [10, 5000, 40000])
def test_zero_direction(vf, ctx, n):
    g = vf.RegularGrid((8, 8, 8), np.zeros(3, np.float32), np.full(3, 8, np.float32), ctx)
    rays = _rays(np.array((8, 8, 8)), n, np.random.default_rng(1))
    rays[n - 2, 3:] = 0.0
    rays[n - 4, 3:] = (0.0, -0.0, 0.0)
    out = np.full((n, 3), 77, np.uint32)
    assert vf.lib().vf_ray_entry_voxels(g.h, vf._p(rays), n, vf._p(out)) != 0
    assert (out == 77).all()
    with pytest.raises(Exception, match=f"ray {n - 4} has a zero direction"):
        g.rayEntryVoxels(rays)
    g.close()
