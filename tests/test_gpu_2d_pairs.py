"""The D2Q9 step kernel steps cell pairs in packed FP32: bit for bit the
oracle's populations where a pair can go wrong (one cell, odd cell counts,
pairs that cross a row end or a tile of 256 cells, a solid partner), and over
enough steps of a full image that a single product contracted into a sum
would show (one ulp in one population was seen after 319 steps)."""
import numpy as np
import pytest

from flow_anizotropy_b200 import solver as S
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _compare(solid, force, nsteps, tau):
    f, u, q = S.debug_steps2d(solid, force, nsteps, tau=tau)
    o = O.State2D(solid, tau)
    o.reset(force)
    o.step(nsteps)
    pore = solid == 0
    assert np.array_equal(f[pore], o.f()[pore])
    assert np.array_equal(u, o.u())
    np.testing.assert_allclose(q, o.q(), rtol=1e-14, atol=1e-30)


@pytest.mark.parametrize("shape", [(1, 1), (1, 2), (2, 1), (3, 3), (1, 255), (1, 257), (3, 85), (17, 31), (128, 4), (5, 513)])
@pytest.mark.parametrize("frac", [0.0, 0.4])
def test_pair_edges(gpu, shape, frac):
    solid = (np.random.default_rng(shape[0] + shape[1]).random(shape) < frac).astype(np.uint8)
    solid.flat[-1] = 0
    for nsteps in (1, 2, 7):
        _compare(solid, [2.5e-7, -1e-7], nsteps, 1.0)


@pytest.mark.parametrize("force", [(2.5e-7, 0.0), (0.0, 2.5e-7), (3e-7, -2e-7)])
@pytest.mark.parametrize("tau", [1.0, 0.995, 0.7])
def test_long_run(gpu, force, tau):
    solid = (np.random.default_rng(4).random((256, 256)) < 0.15).astype(np.uint8)
    _compare(solid, list(force), 700, tau)


def test_many_equal_alone(gpu):
    """A launch of several images, steps whose flags come from the masks and
    from the step itself (lags and averages that cut chunks)."""
    rng = np.random.default_rng(5)
    solids = (rng.random((5, 33, 47)) < 0.25).astype(np.uint8)
    F = 2.5e-7 * np.eye(2)
    p = S.Params2D(tau=0.9, lag=130, hold=2, min_steps=260, max_steps=910, avg_steps=137, avg_sample=13)
    many, _ = S.solve2d_many(solids, F, p)
    for solid, runs in zip(solids, many):
        alone, _, _ = S.solve2d(solid, F, p)
        for a, b, f in zip(runs, alone, F):
            r = O.solve2d(solid, f, tau=0.9, lag=130, hold=2, min_steps=260, max_steps=910, avg_steps=137, avg_sample=13)
            assert (a.steps, a.converged) == (b.steps, b.converged) == (r["steps"], r["converged"])
            assert np.array_equal(a.q, b.q) and np.array_equal(a.se, b.se)
            np.testing.assert_allclose(a.q, r["q"], rtol=1e-12)
