"""A flood with more 256-row units than a CTA keeps a list of (csrc/vf_flood.cu, UNITS: 2048
a CTA, 80 M rows on a whole GPU): 4096 x 4096 x 97 voxels, 84 M rows, empty but for blocks at
the corners, in the middle and across a unit's end, each flooded from seeds of its own.
Every block must equal the oracle's flood of it alone, and the rest stay empty."""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu

SHAPE, BLOCK = (4096, 4096, 97), (24, 30, 37)


@pytest.fixture(scope="module", autouse=True)
def _oracle(oracle_lib):
    return oracle_lib


@pytest.mark.parametrize("dfunc", [1, 2])
def test_unlisted_units(vf, dfunc):
    rng = np.random.default_rng(dfunc)
    occ = np.zeros(SHAPE, np.uint16)
    at = [(0, 0, 0), (4072, 4066, 60), (0, 4066, 31), (4072, 0, 13), (2000, 2040, 20), (1023, 250, 45), (3000, 3333, 60)]
    seeds, want, label = [], [], 2
    for p in at:
        block = (rng.random(BLOCK) < 0.7).astype(np.uint16)
        own = np.argwhere(block)
        own = own[rng.choice(len(own), 5, replace=False)]
        s = np.concatenate([own, np.arange(label, label + 5)[:, None]], axis=1).astype(np.uint32)
        label += 5
        want.append(O.flood(block, s, dfunc)[0])
        seeds.append(s + np.array(list(p) + [0], np.uint32))
        occ[tuple(slice(a, a + b) for a, b in zip(p, BLOCK))] = block
    c = vf.Context(0)
    g = vf.RegularGrid(SHAPE, None, None, c)
    try:
        g.upload(occ)
        fr = vf.FloodFracturer()
        fr.setDistanceFunction(dfunc)
        fr.build(g, np.concatenate(seeds))
        got = g.data()
    finally:
        g.close()
        c.close()
    for p, w in zip(at, want):
        sl = tuple(slice(a, a + b) for a, b in zip(p, BLOCK))
        assert np.array_equal(got[sl], w), p
        got[sl] = 0
    assert not got.any()
