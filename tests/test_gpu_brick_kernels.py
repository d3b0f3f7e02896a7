"""Kernels that deal a brick's voxels to its threads (csrc/vf_gridops.cu) at the
sizes where their rules change: the nearest-seed labelling around its rounds of
seeds, with ties, seeds outside the grid and every seed kept; boundaries where
labels meet at a brick's or window's edge; erosion windows at the grid's ends.
Labels must equal the oracle's bit for bit."""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _oracle(oracle_lib):
    return oracle_lib


def _grid(vf, ctx, lab):
    g = vf.RegularGrid(lab.shape, None, None, ctx)
    g.upload(lab)
    return g


@pytest.mark.parametrize("dfunc", [0, 1, 2])
@pytest.mark.parametrize("shape,nseeds,spread", [
    ((2, 2, 2), 1, 2), ((16, 16, 32), 2, 40), ((17, 33, 31), 255, 33), ((33, 18, 65), 256, 8), ((40, 20, 70), 257, 3),
    ((48, 48, 40), 700, 2), ((20, 20, 100), 4095, 100), ((60, 64, 64), 64, 5000), ((19, 40, 33), 9, 600_000_000)])
def test_nearest_seed(vf, ctx, shape, nseeds, spread, dfunc):
    rng = np.random.default_rng(nseeds + spread)
    occ = (rng.random(shape) < 0.3).astype(np.uint16) * rng.integers(1, 4, shape).astype(np.uint16)
    # the first half within `spread` of the origin (repeats: the lowest index wins), the rest over the grid
    at = rng.integers(0, spread, (nseeds, 3))
    at[nseeds // 2:] = rng.integers(0, shape, (nseeds - nseeds // 2, 3))
    seeds = np.concatenate([at, rng.integers(0, 70000, (nseeds, 1))], axis=1).astype(np.uint32)
    g = _grid(vf, ctx, occ)
    vf.NaiveFracturer().build(g, seeds, vf.Params.default(distance=dfunc))
    assert np.array_equal(g.data(), O.naive(occ, seeds, dfunc))


def _labels(shape, cell, marked, seed):
    """Blocks of one label with empty voxels between; some voxels marked already."""
    rng = np.random.default_rng(seed)
    n = [(s + c - 1) // c for s, c in zip(shape, cell)]
    lab = rng.integers(2, 6, n).astype(np.uint16)
    for a in range(3):
        lab = np.repeat(lab, cell[a], axis=a)
    lab = np.ascontiguousarray(lab[: shape[0], : shape[1], : shape[2]])
    lab[rng.random(shape) < 0.4] = 0
    lab[rng.random(shape) < 0.05] = 1
    lab[(rng.random(shape) < marked) & (lab > 1)] |= 0x8000
    return lab


SHAPES = [((2, 2, 2), (1, 1, 1)), ((16, 16, 32), (16, 16, 32)), ((33, 17, 65), (16, 16, 32)),
          ((40, 50, 70), (17, 15, 34)), ((35, 36, 100), (19, 19, 31)), ((50, 50, 37), (50, 50, 37))]


@pytest.mark.parametrize("bs", [0, 1, 2, 3])
@pytest.mark.parametrize("marked", [0.0, 0.01])
@pytest.mark.parametrize("shape,cell", SHAPES)
def test_boundaries(vf, ctx, shape, cell, marked, bs):
    lab = _labels(shape, cell, marked, 3)
    g = _grid(vf, ctx, lab)
    g.detectBoundaries(bs)
    assert np.array_equal(g.data(), O.detect_boundaries(lab, bs))


@pytest.mark.parametrize("etype,size,iters", [(0, 1, 1), (0, 3, 2), (1, 5, 1), (2, 7, 1), (0, 7, 2), (1, 3, 1)])
@pytest.mark.parametrize("shape,cell", SHAPES)
def test_erosion(vf, ctx, shape, cell, etype, size, iters):
    lab = _labels(shape, cell, 0.0, 5)
    g = _grid(vf, ctx, lab)
    g.erode(etype, size, iters, 0.7, 0.5, 11)
    assert np.array_equal(g.data(), O.erode(lab, etype, size, iters, 0.7, 0.5, 11))


@pytest.mark.parametrize("shape,cell", SHAPES)
def test_isolated(vf, ctx, shape, cell):
    lab = _labels(shape, cell, 0.02, 7)
    g = _grid(vf, ctx, lab)
    g.removeIsolatedRegions()
    assert np.array_equal(g.data(), O.remove_isolated(lab))
