"""Batch chunks that are not a multiple of 4 (the step kernels then take the
lattice of the two-lattice forms from a solve's own step number) and chunks of
several reduction passes, the last one partial.  The first direction of the
structure, which leads its group, ends long before the others (a force so
large that its flux is not finite by the first lag): the others must have the
bits of the same directions solved alone."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", ["fp64", "fp32", "fp16", "bf16"])
@pytest.mark.parametrize("chunk", [6, 64, 100, 128, 130])
def test_chunks(gpu, prec, chunk):
    from flow_anizotropy_b200.solver import Batch, Params3D, solve3d
    solid = (np.random.default_rng(5).random((12, 13, 14)) < 0.35).astype(np.uint8)
    F = np.array([[1e3, 0, 0], [0, 1e-6, 0], [1e-6, 0, -2e-6]])
    p = Params3D(eps=0.0, lag=40, min_steps=80, max_steps=410, avg_steps=33, precision=prec, criterion="drift")
    b = Batch(precision=prec, hbm_budget=2 ** 31, chunk=chunk)
    assert b.submit(solid, F, p, tag=7)
    done = []
    for _ in range(2 + 443 // chunk):
        b.run(1)
        done += b.poll()
    b.close()
    assert len(done) == 1 and done[0][0] == 7
    lead, *others = done[0][1]
    assert lead.status == 2 and lead.steps < 300
    alone, _, _ = solve3d(solid, F[1:], p)
    for x, y in zip(others, alone):
        assert x.steps == y.steps == 443 and x.converged == y.converged
        assert np.array_equal(x.q, y.q) and np.array_equal(x.se, y.se)
