"""The adjoint's end state where a species' particles were never set: they rest at the
origin, as they do when set so, and the other species' results stay in their slots.

Tolerance: the two runs add the same FP64 charges in another order: 1e-9."""
import numpy as np
import pytest

from pic_b200 import Consts, adjoint, workloads

M = 33


@pytest.mark.gpu
@pytest.mark.parametrize("unset", [0, 1])
@pytest.mark.parametrize("n", [(7, 5), (300, 129)])
def test_state_of_a_species_that_was_not_set(n, unset):
    mask, seg = adjoint.wall_segments(M, M)
    sp = [dict(n=k, charge=q, mass=m, np2c=2e6) for k, q, m in
          zip(n, (-Consts.qe, Consts.qe), (Consts.me, workloads.ION_MASS))]
    rng = np.random.default_rng(3)
    given = [rng.uniform(4.0, 28.0, n[1 - unset]) for _ in range(2)] + [rng.normal(0, 1e3, n[1 - unset]) for _ in range(2)]
    states = []
    for explicit in (False, True):
        prob = adjoint.AdjointProblem(M, M, 1e-4, 1e-4, 1e-11, sp, mask, seg, 4, 5, 3, tol=1e-11)
        prob.set_particles(1 - unset, *given)
        if explicit:
            prob.set_particles(unset, *[np.zeros(n[unset])] * 4)
        prob.set_target(adjoint.target_density(M, M, 1e14, 5))
        prob.forward(np.array([20.0, -5.0, 11.0, 3.0]), 0.0)
        states.append([t.cpu().numpy().copy() for t in prob.state()])
    for a, b in zip(*states):
        np.testing.assert_allclose(a, b, rtol=1e-9, atol=1e-9 * max(1.0, np.abs(b.astype(np.float64)).max()))
    at = 0 if unset == 1 else n[0]
    assert np.abs(states[0][0][at:at + n[1 - unset]] - given[0]).max() < 1.0
