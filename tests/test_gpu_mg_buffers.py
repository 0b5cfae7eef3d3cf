"""The buffers a multigrid solver is given: a pair that stays is solved in place, whatever
pair came before it.

Oracle: a solver of its own for each pair, bit for bit.
"""
import time

import numpy as np
import pytest
import torch

from pic_b200.multigrid import MultigridSolver

pytestmark = pytest.mark.gpu
N, DX = 513, 1e-4


def box():
    mask = np.zeros((N, N), np.uint8)
    mask[0] = mask[-1] = mask[:, 0] = mask[:, -1] = 1
    f = torch.randn(N, N, generator=torch.Generator(device="cuda").manual_seed(2), device="cuda",
                    dtype=torch.float64) * 1e6
    f[torch.as_tensor(mask, device="cuda") == 1] = 0
    return mask.reshape(-1), f.reshape(-1)


def test_a_pair_that_stays_costs_no_copies():
    """A converged solve is one pass over the grid: three copies of it would show (1.45 of
    the time at 513^2).  Fastest of 300 calls."""
    mask, f = box()
    done = torch.zeros_like(f)
    MultigridSolver(mask, N, N, DX).solve(done, f, tol=1e-12, max_cycles=30)
    best = []
    for earlier in (False, True):
        mg = MultigridSolver(mask, N, N, DX)
        if earlier:
            mg.solve(torch.zeros_like(f), f.clone(), tol=1e-8)
        best.append(1.0)
        for _ in range(300):
            torch.cuda.synchronize()
            t = time.perf_counter()
            mg.solve(done, f, tol=1e-8)
            best[-1] = min(best[-1], time.perf_counter() - t)
    assert best[1] < 1.2 * best[0], best


@pytest.mark.parametrize("order", ["ABABAB", "ABBBAA", "AABBCCA", "ABCABC"])
def test_any_order_of_pairs(order):
    mask, f = box()
    mg = MultigridSolver(mask, N, N, DX)
    pairs = {k: (torch.zeros_like(f), (f * (i + 1)).clone()) for i, k in enumerate("ABC")}
    for k in order:
        phi, g = pairs[k]
        phi.zero_()
        _, (n, r) = mg.solve(phi, g, tol=1e-8)
        want = torch.zeros_like(f)
        assert MultigridSolver(mask, N, N, DX).solve(want, g, tol=1e-8)[1] == (n, r)
        assert torch.equal(phi, want)
