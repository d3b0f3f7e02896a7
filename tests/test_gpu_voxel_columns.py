"""Voxelizer stages (csrc/vf_voxelize.cu) at the sizes where their splits change:
the parity prefix along x around 16 and 512 cells, vertex counts around the
centroid's strides, closed and open meshes, slice planes at the vertices.  Bit for
bit against the oracle."""
import numpy as np
import pytest

import oracle as O
from voxelfragmentml_gb300 import vessel as Vs

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _oracle(oracle_lib):
    return oracle_lib


def _check(vf, ctx, v, f, dims, mn, mx):
    g = vf.RegularGrid(dims, mn, mx, ctx)
    g.fill(v, f)
    assert np.array_equal(g.data(), O.voxelize(v, f, dims, mn, mx))
    g.close()


@pytest.mark.parametrize("X", [2, 15, 16, 17, 31, 32, 33, 511, 512, 513, 1030])
@pytest.mark.parametrize("rest", [(5, 33), (34, 64)])
@pytest.mark.parametrize("open_faces", [0, 1, 40])
def test_prefix(vf, ctx, X, rest, open_faces):
    v, f = Vs.vessel_mesh(16, 12, 1)
    mn, mx = Vs.mesh_aabb(v)
    _check(vf, ctx, v, f[: len(f) - open_faces], (X,) + rest, mn, mx)


@pytest.mark.parametrize("nverts", [3, 1023, 1024, 1025, 8191, 8192, 8193, 20000])
def test_centroid(vf, ctx, nverts):
    rng = np.random.default_rng(nverts)
    v = rng.normal(size=(nverts, 3)).astype(np.float32) * [1.0, 2.0, 0.5] + 3.0
    v = v.astype(np.float32)
    f = rng.integers(0, nverts, (12, 3)).astype(np.uint32)  # open: the centroid's faces count
    _check(vf, ctx, v, f, (24, 26, 28), v.min(0), v.max(0))


@pytest.mark.parametrize("Y", [2, 3, 64, 100, 4096])
def test_planes(vf, ctx, Y):
    # vertices on and between slice planes, and beyond the box
    t = np.arange(-8, 3 * Y // 2 + 8, max(1, Y // 48), dtype=np.float32) / Y
    v = np.stack([np.tile([0.1, 0.9, 0.4], len(t)), np.repeat(t, 3), np.tile([0.2, 0.3, 0.8], len(t))], 1)
    v = v.astype(np.float32)
    f = np.stack([np.arange(0, len(v) - 5, 2), np.arange(3, len(v) - 2, 2), np.arange(5, len(v), 2)], 1).astype(np.uint32)
    _check(vf, ctx, v, f, (7, Y, 9), np.zeros(3, np.float32), np.ones(3, np.float32))
