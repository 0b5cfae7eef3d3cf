"""A simulation's field solves that need more cycles than its step launches in line: the
rest run in one cooperative launch (k_rt_rest in pic_b200/csrc/mg_regtile.cuh).

With a tolerance that no solve reaches, every step's solve runs to max_cycles, five past
the seven in line.  Small r-z grids are the ones whose cooperative launch has more blocks
(a warp per row of the coarsest solve) than the finest level has tiles, so that the
buffer of the blocks' sums must be sized for it.

Oracle: the number of cycles and the norm that the launch reports, and on Cartesian grids
the FP64 residual of the potential for the density that the step deposited (an r-z density
is rounded to FP32 once more after the solver has taken it).
Tolerance: both residuals at FP64's floor, 1e-9 of ||f|| (a V-cycle divides the residual by
50 or more: the seven cycles alone reach 1e-11).
"""
import numpy as np
import pytest
import torch

from pic_b200 import Consts, _lib
from pic_b200.simulation import PICSimulation

DX, CYCLES = 1e-4, 12


def load(sim):
    rng = np.random.default_rng(1)
    n = sim.species[0]["capacity"]
    for s in (0, 1):
        sim.load(s, rng.uniform(1, sim.nx - 2, n), rng.uniform(1, sim.ny - 2, n),
                 *[rng.normal(0, 1e4, n) for _ in range(3)])
    sim.init()


def make(nx, ny, rz, precision="mixed", sweeps=2):
    mask = np.zeros((ny, nx), np.uint8)
    mask[-1] = mask[:, 0] = mask[:, -1] = 1
    if not rz:
        mask[0] = 1
    n = 20_000
    sp = [dict(name=k, charge=q, mass=m, np2c=1e4, capacity=n)
          for k, q, m in (("e", -Consts.qe, Consts.me), ("i", Consts.qe, 40 * Consts.mp))]
    sim = PICSimulation(nx, ny, DX, DX, 1e-12, sp, mask, tol=1e-300, max_cycles=CYCLES, precision=precision,
                        pre_sweeps=sweeps, post_sweeps=sweeps, use_graph=True, geometry="rz" if rz else "cartesian")
    load(sim)
    return sim, mask


def residual(sim, mask):
    """||f - lap(phi)|| / ||f|| over the free nodes, FP64 on the host."""
    ny, nx = mask.shape
    phi, rho = (a.cpu().numpy().astype(np.float64).reshape(ny, nx) for a in sim.fields()[:2])
    p = np.pad(phi, 1)
    lap = (p[1:-1, :-2] + p[1:-1, 2:] + p[2:, 1:-1] + p[:-2, 1:-1] - 4 * phi) / (DX * DX)
    f, free = -rho / Consts.eps0, mask == 0
    return np.linalg.norm((f - lap)[free]) / np.linalg.norm(f[free])


@pytest.mark.gpu
@pytest.mark.parametrize("sweeps", [1, 2, 3])
@pytest.mark.parametrize("precision", ["mixed", "fp64"])
@pytest.mark.parametrize("shape", [(65, 65, True), (49, 65, True), (65, 49, True), (97, 65, True), (129, 97, True),
                                   (65, 65, False), (129, 97, False), (513, 385, False)])
def test_cycles_past_those_in_line(shape, precision, sweeps):
    nx, ny, rz = shape
    sim, mask = make(nx, ny, rz, precision, sweeps)
    for _ in range(2):
        sim.step(2)
        c = sim.counters()
        assert c["last_cycles"] == CYCLES
        assert c["last_rel_res"] < 1e-9 and (rz or residual(sim, mask) < 1e-9)
    sim.close()


@pytest.mark.gpu
@pytest.mark.parametrize("rz", [False, True])
def test_barrier_timeout_is_reported_and_cleared(rz):
    """With the wait limit lowered to one poll the launch's barriers give up; the error is
    reported once, and the simulation steps as before with the default limit.  (The limit
    is the particle pass's too: one report names both.)"""
    sim, mask = make(129, 97, rz)
    sim.step(1)
    sim.counters()
    sim.set_wait_limit(1)
    sim.step(3)
    said = []
    for _ in range(3):
        try:
            sim.counters()
        except _lib.PicError as e:
            assert e.code == _lib.PIC_ERR_TIMEOUT
            said.append(str(e))
    assert len(said) == 1 and "grid barrier" in said[0], said
    torch.cuda.synchronize()  # the context is intact
    sim.set_wait_limit(-1)
    load(sim)
    sim.step(2)
    c = sim.counters()
    assert c["last_cycles"] == CYCLES and c["last_rel_res"] < 1e-9
    sim.close()
