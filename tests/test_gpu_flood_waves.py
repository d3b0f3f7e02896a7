"""The wave flood (csrc/vf_flood.cu) at the sizes where its layout changes:
words and rows around 32, the plane counts (64 / 65 seeds, more than 1024),
word ends crossed along z, one-CTA gangs and larger ones, more jobs than a gang
takes, more candidate rows than a round lists.  Labels must equal the oracle's
bit for bit."""
import numpy as np
import pytest

import oracle as O
from voxelfragmentml_gb300 import vessel as Vs

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _oracle(oracle_lib):
    return oracle_lib


def _flood(vf, ctx, occ, seeds, dfunc):
    g = vf.RegularGrid(occ.shape, None, None, ctx)
    g.upload(occ)
    fr = vf.FloodFracturer()
    fr.setDistanceFunction(dfunc)
    fr.build(g, seeds)
    out = g.data()
    g.close()
    return out


def _seeds(occ, n, rng):
    at = np.argwhere(occ)
    at = at[np.sort(rng.choice(len(at), min(n, len(at)), replace=False))]
    label = np.arange(len(at)) % 254 + 2  # plain fragment labels
    return np.concatenate([at, label[:, None]], axis=1).astype(np.uint32)


@pytest.mark.parametrize("dfunc", [1, 2])
@pytest.mark.parametrize("shape,frac,nseeds", [
    ((2, 2, 2), 1.0, 2), ((3, 33, 31), 0.6, 5), ((5, 31, 32), 0.55, 64), ((4, 32, 33), 0.6, 65),
    ((33, 7, 65), 0.5, 3), ((2, 65, 200), 0.45, 9), ((40, 3, 129), 0.9, 254), ((17, 64, 64), 0.35, 33),
    ((70, 70, 70), 1.0, 4095), ((64, 60, 96), 0.8, 1025), ((130, 128, 20), 0.5, 64), ((96, 100, 160), 0.4, 40)])
def test_flood_edges(vf, ctx, shape, frac, nseeds, dfunc):
    rng = np.random.default_rng(sum(shape) + nseeds)
    occ = (rng.random(shape) < frac).astype(np.uint16)
    seeds = _seeds(occ, nseeds, rng)
    assert np.array_equal(_flood(vf, ctx, occ, seeds, dfunc), O.flood(occ, seeds, dfunc)[0])


def _check_batch(vf, ctx, sizes):
    specs, wants = [], []
    for i, z in enumerate(sizes):
        v, f = Vs.vessel_mesh(12 + i % 5, 9, i)
        mn, mx = Vs.mesh_aabb(v)
        dims = (max(16, z - i % 7), max(16, z - i % 3), z)
        p = vf.Params.default(distance=i % 3, num_seeds=2 + i % 9, seed=i + 1, seed_location=vf.BOTH)
        specs.append(vf.JobSpec(v, f, p, dims=dims, aabb=(mn, mx), ncounts=256))
        q = O.Params()
        for name, _ in O.Params._fields_:
            setattr(q, name, getattr(p, name))
        wants.append(O.run_job(v, f, dims, mn, mx, q, ncounts=256)[:2])
    for r, s, (lab, cnt) in zip(vf.batch_run(specs, ctx), specs, wants):
        assert r.status == 0
        assert np.array_equal(s.labels, lab) and np.array_equal(s.counts, cnt)


@pytest.mark.parametrize("sizes", [[16, 40, 17, 33], [24, 90, 18, 130, 64], [16] * 270 + [120]],
                         ids=["one_cta_each", "two_gangs", "more_jobs_than_a_gang"])
def test_flood_gangs(vf, ctx, sizes):
    _check_batch(vf, ctx, sizes)


@pytest.mark.parametrize("dfunc", [1, 2])
@pytest.mark.parametrize("shape,frac,nseeds,nfrag,nprefix", [
    ((20, 33, 40), 0.45, 9, 2, 3), ((31, 32, 65), 0.4, 64, 7, 4), ((40, 20, 96), 0.35, 65, 30, 2),
    ((33, 47, 33), 0.6, 300, 5, 100), ((24, 24, 70), 0.3, 1100, 254, 5)])
def test_flood_prefix_sets(vf, ctx, shape, frac, nseeds, nfrag, nprefix, dfunc):
    """Sub-seed prefixes: labels shared by several seeds, seeds on one voxel, fragments
    in several components, at every plane count."""
    rng = np.random.default_rng(sum(shape) + nseeds)
    occ = (rng.random(shape) < frac).astype(np.uint16)
    seeds = _seeds(occ, nseeds, rng)
    n = len(seeds)
    seeds[:, 3] = (rng.integers(0, nfrag, n) + 2) | (rng.integers(0, nprefix, n) << 8)
    seeds[n // 2, :3] = seeds[0, :3]  # the later one holds the voxel
    seeds = seeds[rng.permutation(n)]
    assert np.array_equal(_flood(vf, ctx, occ, seeds, dfunc), O.flood(occ, seeds, dfunc)[0])


def test_flood_prefixes_in_a_batch(vf, ctx):
    # jobs with and without sub-seeds in one batch, in step
    specs, wants = [], []
    for i, (z, extra) in enumerate([(40, 0), (96, 12), (33, 5), (100, 0), (64, 30)]):
        v, f = Vs.vessel_mesh(20, 15, i)
        mn, mx = Vs.mesh_aabb(v)
        p = vf.Params.default(distance=i % 3, num_seeds=4 + i, num_extra_seeds=extra, seed=i + 1)
        specs.append(vf.JobSpec(v, f, p, dims=(z - 3, z, z), aabb=(mn, mx), ncounts=256))
        q = O.Params()
        for name, _ in O.Params._fields_:
            setattr(q, name, getattr(p, name))
        wants.append(O.run_job(v, f, specs[-1].dims, mn, mx, q, ncounts=256)[:2])
    for r, s, (lab, cnt) in zip(vf.batch_run(specs, ctx), specs, wants):
        assert r.status == 0 and np.array_equal(s.labels, lab) and np.array_equal(s.counts, cnt)


def test_labels_dealt_to_resident_blocks(vf, ctx):
    # more live bricks than resident blocks, jobs changing under a block,
    # slot planes in one load and past it, bricks that reach past their grid
    specs, wants = [], []
    for i in range(48):
        v, f = Vs.vessel_mesh(20 + i % 5, 15, i)
        mn, mx = Vs.mesh_aabb(v)
        p = vf.Params.default(distance=i % 3, num_seeds=(3, 64, 65, 200)[i % 4], seed=i + 1, seed_location=vf.BOTH,
                              num_extra_seeds=400 if i % 3 == 2 and i % 4 else 0)
        specs.append(vf.JobSpec(v, f, p, dims=(113 + i % 4, 97 + i % 9, 96 + i), aabb=(mn, mx), ncounts=256))
        q = O.Params()
        for name, _ in O.Params._fields_:
            setattr(q, name, getattr(p, name))
        wants.append(O.run_job(v, f, specs[-1].dims, mn, mx, q, ncounts=256)[:2])
    for r, s, (lab, cnt) in zip(vf.batch_run(specs, ctx), specs, wants):
        assert r.status == 0 and np.array_equal(s.labels, lab) and np.array_equal(s.counts, cnt)
