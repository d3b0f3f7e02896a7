"""Point clouds (csrc/vf_sample.cu) where the area sums and the face draws change
their path: chunks of 1024 faces, areas of one size and over a range no double sum
is exact for, areas that are not finite, draws with many repeats.  Bit for bit
against the oracle."""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _oracle(oracle_lib):
    return oracle_lib


def _check(vf, ctx, v, f, S, seed):
    v = v.astype(np.float32)
    f = f.astype(np.uint32)
    got = vf.sample_mesh(v, f, S, seed, ctx)
    v4 = np.concatenate([v, np.zeros((len(v), 1), np.float32)], 1)
    f4 = np.concatenate([f, np.zeros((len(f), 1), np.uint32)], 1)
    e = O.sample_mesh(v4, f4, S, seed, 0)
    assert np.array_equal(got.view(np.uint32), e.view(np.uint32))


@pytest.mark.parametrize("T", [1, 31, 32, 1023, 1024, 1025, 5000])
@pytest.mark.parametrize("spread", [0.0, 3.0, 8.0, 30.0])
def test_sums(vf, ctx, T, spread):
    rng = np.random.default_rng(T)
    v = rng.normal(size=(3 * T, 3)) * np.repeat(2.0 ** (rng.normal(size=T) * spread / 2), 3)[:, None]
    f = np.arange(3 * T).reshape(T, 3)
    f[:: 7] = 0  # areas of zero
    for S in (T + 1, 2 * T + 40):
        _check(vf, ctx, v, f, S, 5)


@pytest.mark.parametrize("bad", [1e30, 1e-30, np.inf])
def test_not_finite(vf, ctx, bad):
    rng = np.random.default_rng(1)
    v = rng.normal(size=(300, 3))
    v[17] = bad
    f = rng.integers(0, 300, (900, 3))
    f[450:] = [1, 2, 3]
    _check(vf, ctx, v, f, 400, 3)


@pytest.mark.parametrize("T,S", [(1, 1), (2, 2), (255, 255), (256, 200), (257, 257), (3000, 2999), (70000, 1024)])
def test_draws(vf, ctx, T, S):
    rng = np.random.default_rng(S)
    v = rng.normal(size=(100, 3))
    _check(vf, ctx, v, rng.integers(0, 100, (T, 3)), S, 11)
