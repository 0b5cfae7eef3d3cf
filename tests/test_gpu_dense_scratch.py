"""The dense deposit and gather where their scratch does not fit on the device: the plain
operators do the same work without it.

Oracle: the same calls with the scratch; tolerance of the density as in test_gpu_dense_ops,
the velocities bit for bit."""
import numpy as np
import pytest
import torch

from pic_b200 import Consts, Grid
from pic_b200.Particles import Particles2D


def full(*args, **kwargs):
    raise torch.OutOfMemoryError("no room")


@pytest.mark.gpu
def test_no_room_for_the_scratch(monkeypatch):
    m, nn, n = 65, 33, 20_000
    monkeypatch.setattr(Grid, "DENSE_PARTICLES", 0)
    out = []
    for room in (True, False):
        grid = Grid.Grid2D(m, nn, 1e-4 * (m - 1), 1e-4 * (nn - 1))
        parts = Particles2D(n)
        parts.grid, parts.np2c = grid, 1e4
        parts.add_species("e", Consts.me, -Consts.qe, 0)
        rng = np.random.default_rng(1)
        parts.load_species_arrays(1, rng.uniform(0, grid.X, n), rng.uniform(0, grid.Y, n), rng.normal(0, 1e5, n),
                                  rng.normal(0, 1e5, n))
        grid.E.copy_(torch.as_tensor(rng.normal(0, 1e3, (2, m * nn)).astype(np.float32), device="cuda"))
        with monkeypatch.context() as c:
            if not room:
                c.setattr(torch, "empty", full)
            grid.update_density(parts)
            parts.update_V(grid, 1e-11)
        assert (grid._cells is not None) == room and (grid._pairs is not None) == room
        s = parts.species[0]
        out.append((grid.rho.cpu(), s.vx.cpu(), s.vy.cpu()))
    (r0, *v0), (r1, *v1) = out
    assert (r0 - r1).abs().max() <= 1e-5 * r0.abs().max()
    for a, b in zip(v0, v1):
        assert torch.equal(a.view(torch.int32), b.view(torch.int32))
