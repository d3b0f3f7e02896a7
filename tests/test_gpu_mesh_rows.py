"""Fragment meshes at the sizes where the packed row kernels and the smoothing
lists (csrc/vf_mesh.cu) change: rows around 8, 16, 256 and 512 voxels, 255 to 257
fragments, vertices with many faces, chunks of 256 vertices.  Bit for bit against
the oracle."""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _oracle(oracle_lib):
    return oracle_lib


def _check(vf, ctx, lab, p):
    mn, mx = np.array([-1.5, 0.25, -3.0], np.float32), np.array([2.0, 1.75, 5.5], np.float32)
    g = vf.RegularGrid(lab.shape, mn, mx, ctx)
    g.upload(lab)
    sizes = g.triangulate(p)
    vals, vo, fo, v, f = g.meshes_arrays()
    counters = g.mesh_counters()
    g.close()
    e = O.triangulate(lab, mn, mx, p.nonboundary_iterations, p.nonboundary_weight, p.boundary_iterations,
                      p.boundary_weight)
    assert sizes == (len(e[0]), len(e[3]), len(e[4]))
    assert np.array_equal(vals, e[0]) and np.array_equal(vo, e[1]) and np.array_equal(fo, e[2])
    assert np.array_equal(f, e[4])
    assert np.array_equal(v.view(np.uint32), e[3].view(np.uint32))
    return counters


@pytest.mark.parametrize("Z", [2, 7, 8, 15, 16, 17, 255, 256, 257, 511, 512, 513, 530])
@pytest.mark.parametrize("empty,marked", [(0.0, 0.3), (0.6, 0.05), (0.98, 0.5)])
def test_rows(vf, ctx, Z, empty, marked):
    rng = np.random.default_rng(Z)
    lab = rng.integers(0, 6, (4, 3, Z)).astype(np.uint16)
    lab[rng.random(lab.shape) < empty] = 0
    lab[-1, -1, -1] = 5
    lab |= (rng.random(lab.shape) < marked).astype(np.uint16) << 15
    _check(vf, ctx, lab, vf.MCParams(2, 0.7, 3, 0.3))


@pytest.mark.parametrize("values", [1, 254, 255, 256, 257])
def test_fragments(vf, ctx, values):
    rng = np.random.default_rng(values)
    lab = rng.integers(2, 2 + values, (12, 13, 14)).astype(np.uint16)
    lab.ravel()[:values] = np.arange(2, 2 + values)
    _check(vf, ctx, lab, vf.MCParams(1, 0.9, 1, 0.2))


@pytest.mark.parametrize("marked", [0.0, 1.0, 0.01])
def test_passes(vf, ctx, marked):
    # blocks of two fragments: every vertex in one pass, in the other, in both
    rng = np.random.default_rng(3)
    lab = np.ones((30, 41, 50), np.uint16)
    lab[3:28, 4:39, 5:30] = 2
    lab[3:28, 4:39, 30:47] = 3
    lab |= (rng.random(lab.shape) < marked).astype(np.uint16) << 15
    V, T, nb, inc, ent, bent = _check(vf, ctx, lab, vf.MCParams(4, 0.9, 4, 0.2))
    assert (nb == 0) == (marked == 0.0) and nb <= V and bent <= ent <= 2 * inc
