"""V-cycles of more sweeps than the multigrid's register tiles take (four to eight, on
shared-memory tiles), and of such a number on one side only, where one kind of tile hands
over to the other, single levels and two levels per launch alike.

Oracle and tolerances as in test_gpu_mg_regtile: one and three FP64 cycles against
whole-level numpy phases to 1e-12 of max|phi|; one FP32 cycle to 2e-5 of it.
"""
import numpy as np
import pytest
import torch

import test_gpu_mg_regtile as whole
from pic_b200.multigrid import MultigridSolver

pytestmark = pytest.mark.gpu
SWEEPS = [(4, 4), (2, 4), (4, 2), (2, 5), (6, 3), (8, 8)]


@pytest.mark.parametrize("sw", SWEEPS)
@pytest.mark.parametrize("rz", [False, True])
@pytest.mark.parametrize("shape", [(57, 41), (105, 113), (257, 145)])
def test_cycles_against_whole_level_phases(shape, rz, sw):
    whole.test_cycles_against_whole_level_phases(shape, rz, sw)


@pytest.mark.parametrize("sw", SWEEPS)
@pytest.mark.parametrize("rz", [False, True])
@pytest.mark.parametrize("shape", [(105, 113), (257, 145)])
def test_mixed_cycle_against_whole_level_phases(shape, rz, sw):
    nx, ny = shape
    free, phi0, f = whole.problem(nx, ny, rz, electrode=True)
    W = whole.weights(ny, whole.DX, whole.DY, rz)
    mg = MultigridSolver((~free).astype(np.uint8).reshape(-1), nx, ny, whole.DX, omega=whole.OMEGA, precision="mixed",
                         hy=whole.DY, pre_sweeps=sw[0], post_sweeps=sw[1], geometry="rz" if rz else "cartesian")
    r = np.where(free, f - (whole.neighbours(phi0, *W[:3]) - W[3][:, None] * phi0), 0.0)
    want = phi0 + whole.vcycle(r, free, whole.DX, whole.DY, rz, *sw)
    phi = torch.as_tensor(phi0.reshape(-1).copy(), device="cuda")
    mg.solve(phi, torch.as_tensor(f.reshape(-1), device="cuda"), tol=1e-300, max_cycles=1)
    np.testing.assert_allclose(phi.cpu().numpy().reshape(ny, nx), want, rtol=0, atol=2e-5 * np.abs(want).max())
