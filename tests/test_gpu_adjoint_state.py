"""The adjoint's particles: a species that was never set rests at the origin, as it does
when set so, and the other species' results stay in their slots; species set on streams
of their own.

Tolerance: two runs add the same FP64 charges in another order: 1e-9."""
import numpy as np
import pytest
import torch

from pic_b200 import Consts, _lib, adjoint, workloads

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


@pytest.mark.gpu
def test_species_set_on_two_streams():
    """Both species set back to back on streams of their own, the host waiting for neither:
    the same as one after the other (their sorts share scratch)."""
    n = (150_000, 110_003)
    mask, seg = adjoint.wall_segments(M, M)
    sp = [dict(n=k, charge=q, mass=m, np2c=2e3) for k, q, m in
          zip(n, (-Consts.qe, Consts.qe), (Consts.me, workloads.ION_MASS))]
    g = torch.Generator(device="cuda").manual_seed(1)
    parts = [[torch.rand(k, generator=g, device="cuda", dtype=torch.float64) * (M - 1) for _ in range(2)] +
             [torch.randn(k, generator=g, device="cuda", dtype=torch.float64) * 1e3 for _ in range(2)] for k in n]
    states, streams = [], [torch.cuda.Stream() for _ in n]
    for together in (False, True):
        prob = adjoint.AdjointProblem(M, M, 1e-4, 1e-4, 1e-11, sp, mask, seg, 4, 2, 2, tol=1e-11)
        torch.cuda.synchronize()
        for _ in range(3):
            for s, p in enumerate(parts):
                if together:
                    _lib.call("pic_adj_set_particles", prob._h, s, *[_lib.ptr(a) for a in p], None, None,
                              streams[s].cuda_stream)
                else:
                    prob.set_particles(s, *p)
        torch.cuda.synchronize()
        prob.set_target(adjoint.target_density(M, M, 1e14, 5))
        prob.forward(np.zeros(4), 0.0)
        states.append([t.cpu().numpy().copy() for t in prob.state()])
    for a, b in zip(*states):
        np.testing.assert_allclose(a, b, rtol=1e-9, atol=1e-9 * max(1.0, np.abs(b.astype(np.float64)).max()))
