"""The adjoint's particle passes: four slots per thread in cell order, results in the
caller's order.

Particle counts around the four slots and the warp (1 to 1001, different per
species), positions on edges and corners, every particle in one cell (the warp adds
up all its lanes) and spread over the grid (it adds up none): the loss and the end
state against the FP64 CPU restatement, the state in the order the particles were
given in, the gradients unchanged when the particles are given in another order,
and a second backward pass equal to the first.

Tolerances: the forward pass against the restatement as in test_gpu_adjoint (1e-9,
1e-8 cells); another order changes FP64 sums of n terms by about n * 2^-53 of their
largest, and the solves stop at 1e-11: 1e-9 of the largest gradient.
"""
import numpy as np
import pytest
import torch

from oracle import adjoint_ref
from pic_b200 import Consts, adjoint, workloads

pytestmark = pytest.mark.gpu
M, STEPS, EVERY = 33, 7, 3


def problem(parts, steps=STEPS):
    mask, seg = adjoint.wall_segments(M, M)
    sp = [dict(n=p[0].size, charge=q, mass=m, np2c=2e6) for p, q, m in
          zip(parts, (-Consts.qe, Consts.qe), (Consts.me, workloads.ION_MASS))]
    prob = adjoint.AdjointProblem(M, M, 1e-4, 1e-4, 1e-11, sp, mask, seg, 4, steps, EVERY, tol=1e-11)
    for s, (x, y, vx, vy, dv) in enumerate(parts):
        prob.set_particles(s, x, y, vx, vy, dv, 0.5 * dv)
    target = adjoint.target_density(M, M, 1e14, 5)
    prob.set_target(target)
    return prob, sp, mask, seg, target


def species(rng, n, one_cell, vth):
    lo, hi = (7.25, 7.75) if one_cell else (0.0, M - 1.0)
    x, y = rng.uniform(lo, hi, (2, n))
    if not one_cell and n > 8:
        x[:4], y[:4] = [0.0, M - 1.0, M - 1.0, 0.0], [0.0, M - 1.0, 0.0, M - 1.0]
    v = rng.normal(0.0, vth, (2, n))
    return x, y, v[0], v[1], rng.normal(size=n)


@pytest.mark.parametrize("n_e,n_i,one_cell", [(1, 3, False), (5, 2, True), (127, 130, True), (128, 33, False),
                                              (1001, 999, False), (1001, 514, True)])
def test_any_count_and_order(n_e, n_i, one_cell):
    rng = np.random.default_rng(n_e * 7 + n_i)
    parts = [species(rng, n_e, one_cell, 8e5), species(rng, n_i, one_cell, 3e2)]
    V, A = np.array([20.0, -5.0, 11.0, 3.0]), 2e4
    prob, sp, mask, seg, target = problem(parts)
    loss = prob.forward(V, A)
    state = [t.cpu().numpy().copy() for t in prob.state()]
    dV, dA = prob.backward()
    dV2, dA2 = prob.backward()
    scale = np.abs(dV).max()
    assert np.abs(dV2 - dV).max() <= 1e-12 * scale and abs(dA2 - dA) <= 1e-12 * abs(dA)
    ref = adjoint_ref.RefDifferentiable(
        M, M, 1e-4, 1e-4, 1e-11, Consts.eps0,
        [dict(charge=d["charge"], mass=d["mass"], np2c=d["np2c"], x=p[0], y=p[1], vx=p[2], vy=p[3], dvx=p[4],
              dvy=0.5 * p[4]) for d, p in zip(sp, parts)], mask, seg, 4, STEPS, 0, target)
    rloss, pos, alive = ref.run(V, A)
    assert loss == pytest.approx(rloss, rel=1e-9)
    at = 0
    for s, p in enumerate(parts):
        n = p[0].size
        live = np.asarray(alive[s], bool)
        np.testing.assert_array_equal(state[4][at:at + n] > STEPS, live)
        for got, want in zip(state[:2], pos[s]):
            np.testing.assert_allclose(got[at:at + n][live], np.asarray(want)[live], rtol=0, atol=1e-8)
        at += n
    orders = [rng.permutation(p[0].size) for p in parts]
    shuffled, *_ = problem([tuple(a[o] for a in p) for p, o in zip(parts, orders)])
    assert shuffled.forward(V, A) == pytest.approx(loss, rel=1e-12)
    at = 0
    moved = [t.cpu().numpy() for t in shuffled.state()]
    for p, o in zip(parts, orders):
        n = p[0].size
        for a, b in zip(state[:5], moved[:5]):
            np.testing.assert_allclose(b[at:at + n], a[at:at + n][o], rtol=1e-9, atol=1e-9)
        at += n
    sV, sA = shuffled.backward()
    assert np.abs(sV - dV).max() <= 1e-9 * scale and abs(sA - dA) <= 1e-9 * abs(dA)
