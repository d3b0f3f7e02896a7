"""The shell's per-face forms (csrc/vf_voxelize.cu, k_shell_flat) where their
margins decide: triangles on cell boundaries, with edges along the axes, slivers,
far larger or smaller than a cell, beyond the grid, and far from the origin.
Occupancy must equal the oracle's bit for bit."""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _oracle(oracle_lib):
    return oracle_lib


def _soup(kind, n, dims, rng):
    """Triangles of a kind in cell units: [n, 3, 3]."""
    d = np.array(dims, np.float64)
    at = rng.random((n, 1, 3)) * d
    size = {"cells": 3.0, "grid": 4.0, "axes": 9.0, "sliver": 20.0, "huge": 300.0, "tiny": 0.02, "beyond": 60.0,
            "plates": 12.0}[kind]
    t = at + rng.normal(size=(n, 3, 3)) * size
    if kind == "grid":
        t = np.round(t * 2) / 2
    if kind == "axes":  # edges along one axis or another
        t[:, 1, :2] = t[:, 0, :2]
        t[:, 2, 1:] = t[:, 0, 1:]
    if kind == "sliver":
        t[:, 2] = 0.5 * (t[:, 0] + t[:, 1]) + rng.normal(size=(n, 3)) * 0.003
    if kind == "plates":  # planes on and between cell boundaries
        axis = rng.integers(0, 3, n)
        for a in range(3):
            t[axis == a, :, a] = np.round(t[axis == a, :1, a] * 2) / 2
    return t


@pytest.mark.parametrize("offset", [0.0, 40.0, 5000.0])
@pytest.mark.parametrize("kind", ["cells", "grid", "axes", "sliver", "huge", "tiny", "beyond", "plates"])
@pytest.mark.parametrize("dims", [(70, 65, 90), (2, 9, 33), (20, 200, 31)])
def test_shell(vf, ctx, dims, kind, offset):
    rng = np.random.default_rng(len(kind) * 131 + dims[0])
    n = 1 if kind == "huge" and dims[0] < 10 else 90
    cell = np.array([0.011, 0.02, 0.0147])  # metres per cell
    v = (_soup(kind, n, dims, rng) * cell + offset).reshape(-1, 3).astype(np.float32)
    f = np.arange(3 * n, dtype=np.uint32).reshape(n, 3)
    mn = np.full(3, offset, np.float32)
    mx = (np.array(dims) * cell + offset).astype(np.float32)
    g = vf.RegularGrid(dims, mn, mx, ctx)
    g.fill(v, f)
    want = O.voxelize(v, f, dims, mn, mx)
    assert np.array_equal(g.data() != 0, want != 0)
    g.close()
