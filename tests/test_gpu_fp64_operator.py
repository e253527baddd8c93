"""The FP64 collision operator against the CPU oracle, bit for bit, where its
shared products and its quotients by a reciprocal could go wrong: relaxation
times from the stability limit upward (tau = 1 is its own specialisation),
forces along and across the axes, none at all, and velocities far beyond a
solve's, over enough steps that every population has moved."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tau", [0.505, 0.6, 1.0, 2.7])
@pytest.mark.parametrize("force", [(1e-6, 0, 0), (0, 0, -3e-4), (2e-4, -1e-4, 3e-5), (0, 0, 0)])
def test_operator_bitwise(gpu, tau, force):
    from flow_anizotropy_b200.solver import debug_steps3d
    solid = (np.random.default_rng(11).random((7, 9, 33)) < 0.3).astype(np.uint8)
    solid.flat[0] = 0
    f, _, _ = debug_steps3d(solid, force, 25, tau=tau, precision="fp64")
    o = O.State3D(solid, tau)
    o.reset(list(force))
    o.step(25)
    pore = solid == 0
    assert np.array_equal(f[pore], o.f()[pore])
