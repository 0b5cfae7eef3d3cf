"""Which gather Particles2D.update_V takes: the planes for particles that were sorted and
have moved little since, node pairs for any others; the same velocities bit for bit."""
import numpy as np
import pytest
import torch

from pic_b200 import Consts, Grid, Particles, _lib

pytestmark = pytest.mark.gpu


def test_gather_follows_the_order(monkeypatch):
    monkeypatch.setattr(Grid, "DENSE_PARTICLES", 0)
    m, n, rng = 65, 20_000, np.random.default_rng(1)
    grid = Grid.Grid2D(m, m, 1e-4 * (m - 1), 1e-4 * (m - 1))
    parts = Particles.Particles2D(2 * n)
    parts.grid, parts.np2c = grid, 1e4
    parts.add_species("e", Consts.me, -Consts.qe, 0)
    new = lambda: (rng.uniform(0, grid.X, n), rng.uniform(0, grid.Y, n), *rng.normal(0, 1e3, (2, n)))  # noqa: E731
    parts.load_species_arrays(1, *new())
    grid.E.copy_(torch.as_tensor(rng.normal(0, 1e3, (2, m * m)).astype(np.float32), device="cuda"))

    def kick():
        grid._pairs = None
        s = parts.species[0]
        v = [a.clone() for a in (s.vx, s.vy)]
        _lib.call("pic_update_V", _lib.ptr(s.x), _lib.ptr(s.y), _lib.ptr(v[0]), _lib.ptr(v[1]), s.n,
                  _lib.ptr(grid.E[0]), _lib.ptr(grid.E[1]), m, m, float(s.charge / s.mass * 1e-11), _lib.stream_ptr())
        parts.update_V(grid, 1e-11)
        for a, b in zip(v, (s.vx, s.vy)):
            assert torch.equal(a.view(torch.int32), b.view(torch.int32))
        return grid._pairs is not None

    assert kick()
    parts.sort()
    assert not kick()
    for k in range(Particles.SORTED_MOVES):
        parts.update_R(1e-12)
    assert not kick()
    parts.update_R(1e-12)
    assert kick()
    parts.sort()
    assert not kick()
    parts.load_species_arrays(1, *(a[:100] for a in new()))
    assert kick()
