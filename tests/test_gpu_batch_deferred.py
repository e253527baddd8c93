"""A batch makes its work list and graph once before a chunk, not at every
admission: results must not depend on how admissions, polls and runs
interleave (several admissions before a run, polls before any run, slots
freed and taken again, and in FP64, whose operator gives the same bits for
tau = 1 in both of its forms, a relaxation time that changes the kernels
midway)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _solid(n, seed):
    s = (np.random.default_rng(seed).random((n, n + 1, n + 3)) < 0.35).astype(np.uint8)
    s.flat[0] = 0
    return s


@pytest.mark.parametrize("prec", ["fp64", "fp32", "fp16"])
def test_interleaved_admissions(gpu, prec):
    from flow_anizotropy_b200.solver import Batch, Params3D, solve3d
    F = 1e-6 * np.eye(3)

    def params(k):
        return Params3D(tau=0.8 if prec == "fp64" and k >= 4 else 1.0, eps=1e-9, lag=50, min_steps=100, max_steps=100 + 50 * k, avg_steps=40,
                        precision=prec)

    b = Batch(precision=prec, hbm_budget=2 ** 31, chunk=64)
    done = {}
    assert b.poll() == [] and b.active() == 0
    for k in range(3):
        assert b.submit(_solid(10 + k, k), F, params(k), tag=k)
    assert b.active() == 9 and b.poll() == []
    b.run(2)
    for k in range(3, 7):
        assert b.submit(_solid(10 + k, k), F, params(k), tag=k)
        done.update(b.poll())                 # retires some, frees their slots
    for _ in range(40):
        b.run(1)
        done.update(b.poll())
        if len(done) == 7:
            break
    assert b.active() == 0 and b.resident_bytes() == 0
    for k in range(7):
        alone, _, _ = solve3d(_solid(10 + k, k), F, params(k))
        for x, y in zip(done[k], alone):
            assert (x.steps, x.converged) == (y.steps, y.converged)
            assert np.array_equal(x.q, y.q) and np.array_equal(x.se, y.se)
    b.close()
