"""The early-starting step kernels (csrc/step3d_slots.cuh), which the default
variants run, against the work-list kernels of another variant: fluxes,
standard errors, step counts and velocities must have the same bits.  Sizes
are the edges of their dispatch: a single pore, tiles of 511 / 512 / 513
pores, several launches per step (5 directions), tile counts either side of
the split limits (444 tiles for the pull form, 8192 for the others), and step
counts that mix single launches, graph chunks and averaging."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

OTHER = {"fp64": 1, "fp32": 3, "fp16": 0, "bf16": 85}


def _pores(n, shape, seed=0):
    """A mask of `shape` with exactly n pores."""
    solid = np.ones(shape, np.uint8).ravel()
    solid[np.random.default_rng(seed).permutation(solid.size)[:n]] = 0
    return solid.reshape(shape)


def _compare(solid, prec, ndir, tau=1.0, steps=(150, 40), velocity=True):
    from flow_anizotropy_b200.solver import Params3D, solve3d
    F = 1e-6 * np.array([[1, 0, 0], [0, 1, 0], [0, 0, 1], [1, 1, 1], [1, -2, 0.5]])[:ndir]
    p = dict(tau=tau, eps=1e-9, lag=30, min_steps=60, max_steps=steps[0], avg_steps=steps[1], precision=prec)
    a, _, va = solve3d(solid, F, Params3D(**p), velocity=velocity)
    b, _, vb = solve3d(solid, F, Params3D(**p, variant=OTHER[prec]), velocity=velocity)
    for x, y in zip(a, b):
        assert (x.steps, x.converged) == (y.steps, y.converged)
        assert np.array_equal(x.q, y.q) and np.array_equal(x.se, y.se)
    if velocity:
        assert np.array_equal(va, vb)


@pytest.mark.parametrize("prec", ["fp64", "fp32", "fp16", "bf16"])
@pytest.mark.parametrize("n", [1, 511, 512, 513, 1100])
def test_tile_edges(gpu, prec, n):
    _compare(_pores(n, (9, 11, 33), n), prec, 3)


@pytest.mark.parametrize("prec", ["fp64", "fp32", "bf16"])
@pytest.mark.parametrize("ndir,tau", [(1, 0.8), (4, 1.0), (5, 0.8)])
def test_directions(gpu, prec, ndir, tau):
    _compare(_pores(2000, (16, 17, 19), ndir), prec, ndir, tau)


@pytest.mark.parametrize("prec,n", [("fp32", 444 * 512), ("fp32", 444 * 512 + 1), ("fp64", 8192 * 512), ("fp64", 8192 * 512 + 1),
                                    ("bf16", 8192 * 512 + 1)])
def test_split_limits(gpu, prec, n):
    edge = int(np.ceil((n / 0.95) ** (1 / 3)))
    _compare(_pores(n, (edge, edge, edge)), prec, 1, steps=(20, 12), velocity=False)


@pytest.mark.parametrize("prec,n", [("fp64", 45 ** 3), ("fp64", 72 ** 3), ("fp64", 84 ** 3), ("fp32", 64 ** 3), ("fp32", 92 ** 3)])
def test_direction_groups(gpu, prec, n):
    """Lattices of a direction from a few MB to beyond L2: all directions in a
    step, two of three (or of four), one at a time."""
    edge = int(np.ceil((n / 0.8) ** (1 / 3)))
    for ndir in (3, 4):
        _compare(_pores(n, (edge, edge, edge)), prec, ndir, steps=(150, 33), velocity=False)


@pytest.mark.parametrize("n", [166666, 166667])
def test_small_16bit_limit(gpu, n):
    _compare(_pores(n, (60, 60, 60)), "fp16", 3, steps=(70, 20))


@pytest.mark.parametrize("steps", [(1, 0), (3, 2), (64, 0), (129, 1), (130, 64), (259, 130)])
def test_step_counts(gpu, steps):
    _compare(_pores(900, (9, 11, 33), 3), "fp16", 3, steps=steps)
    _compare(_pores(900, (9, 11, 33), 3), "fp64", 2, steps=steps)
