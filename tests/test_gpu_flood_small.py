"""Floods of few rows (csrc/vf_flood.cu): a gang of several CTAs, or its first CTA alone
where at most 48 k voxels are occupied; the gangs of a batch side by side, narrower the
more there are.  Either side of each limit, full and ragged, against the oracle."""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu

LONE = 48 << 10


@pytest.fixture(scope="module", autouse=True)
def _oracle(oracle_lib):
    return oracle_lib


def _occupancy(shape, voxels):
    """The first `voxels` in the grid's order."""
    occ = np.zeros(int(np.prod(shape)), np.uint16)
    occ[:voxels] = 1
    return occ.reshape(shape)


def _seeds(occ, n, rng):
    at = np.argwhere(occ)
    at = at[np.sort(rng.choice(len(at), n, replace=False))]
    return np.concatenate([at, np.arange(2, n + 2)[:, None]], axis=1).astype(np.uint32)


# rows: 62 x 62 x 64 voxels 12162, 72 x 72 x 64 16282, 73 x 73 x 64 16727 (past the limit of small ones)
@pytest.mark.parametrize("dfunc", [1, 2])
@pytest.mark.parametrize("shape,voxels", [
    ((62, 62, 64), LONE), ((62, 62, 64), LONE + 1), ((62, 62, 64), 62 * 62 * 64), ((33, 30, 31), 33 * 30 * 31),
    ((72, 72, 64), LONE), ((72, 72, 64), 72 * 72 * 64), ((73, 73, 64), 73 * 73 * 64), ((16, 16, 16), 4096)])
def test_one_cta_or_several(vf, ctx, shape, voxels, dfunc):
    rng = np.random.default_rng(voxels)
    occ = _occupancy(shape, voxels)
    seeds = _seeds(occ, 5, rng)
    want = O.flood(occ, seeds, dfunc)[0]
    g = vf.RegularGrid(shape, None, None, ctx)
    g.upload(occ)
    fr = vf.FloodFracturer()
    fr.setDistanceFunction(dfunc)
    fr.build(g, seeds)
    got = g.data()
    g.close()
    assert np.array_equal(got, want)
    import torch
    d_occ, d_seeds = torch.from_numpy(occ.view(np.int16)).cuda(), torch.from_numpy(seeds.view(np.int32)).cuda()
    d_lab = torch.zeros_like(d_occ)
    st = vf.lib().vf_flood_noalloc(vf.C.c_void_p(d_occ.data_ptr()), vf.C.c_void_p(d_lab.data_ptr()), *shape,
                                   vf.C.c_void_p(d_seeds.data_ptr()), len(seeds), dfunc, None)
    assert st == 0
    assert np.array_equal(d_lab.cpu().numpy().view(np.uint16), want)


BOX_V = np.array([[x, y, z] for x in (0, 1) for y in (0, 1) for z in (0, 1)], np.float32)
BOX_F = np.array([[0, 1, 3], [0, 3, 2], [4, 6, 7], [4, 7, 5], [0, 4, 5], [0, 5, 1], [2, 3, 7], [2, 7, 6],
                  [0, 2, 6], [0, 6, 4], [1, 5, 7], [1, 7, 3]], np.uint32)


@pytest.mark.parametrize("jobs", [2, 5, 60, 320])  # CTAs enough for full gangs, for narrow ones, for one each
def test_batch_of_small_solids(vf, ctx, jobs):
    """Solid boxes (every voxel) and slabs of one, in a batch where every flood is small."""
    specs = []
    for i in range(jobs):
        z = (64, 40, 17, 50)[i % 4]
        dims = (z - i % 3, z - 1, z)
        p = vf.Params.default(distance=i % 3, num_seeds=2 + i % 5, seed=i + 1, seed_location=vf.BOTH)
        hi = (1.0, 1.0, 1.0) if i % 5 else (1.0, 1.0, 6.0)  # a sixth of the grid
        specs.append(vf.JobSpec(BOX_V, BOX_F, p, dims=dims, aabb=((0.0, 0.0, 0.0), hi), ncounts=256))
    res = vf.batch_run(specs, ctx)
    for r, s in zip(res, specs):
        assert r.status == 0
    for s in specs[:4] + specs[-4:]:
        q = O.Params()
        for name, _ in O.Params._fields_:
            setattr(q, name, getattr(s.params, name))
        lab, cnt = O.run_job(s.verts, s.faces, s.dims, s.aabb[0], s.aabb[1], q, ncounts=256)[:2]
        assert np.array_equal(s.labels, lab) and np.array_equal(s.counts, cnt)
