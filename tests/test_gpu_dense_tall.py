"""The dense deposit and gather on grids of more rows than a launch has blocks in y (65535),
which the plain operators take.

Oracle: FP64 sums of the same weights on the host's side (torch on the GPU), and
pic_update_V, bit for bit.  Tolerance: a node's corner sums are FP32 sums of about two
particles' weights each: 1e-5 of the largest.
"""
import pytest
import torch

from pic_b200 import Consts, _lib
from pic_b200.Grid import Grid2D
from pic_b200.Particles import Particles2D

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,nn", [(3, 70_001), (2, 131_073), (3, 65_536)])
def test_tall_grid(m, nn):
    n = 600_000
    grid = Grid2D(m, nn, 1e-4 * (m - 1), 1e-4 * (nn - 1))
    parts = Particles2D(n)
    parts.grid, parts.np2c = grid, 1e4
    parts.add_species("e", Consts.me, -Consts.qe, 0)
    g = torch.Generator(device="cuda").manual_seed(1)
    r = lambda: torch.rand(n, generator=g, device="cuda", dtype=torch.float64)  # noqa: E731
    parts.load_species_arrays(1, r() * grid.X, r() * grid.Y, r() * 1e5, r() * 1e5)
    s = parts.species[0]
    grid.update_density(parts)
    assert grid._cells is not None
    x, y = s.x[: s.n].double(), s.y[: s.n].double()
    i, j = x.floor().clamp(max=m - 2), y.floor().clamp(max=nn - 2)
    want = torch.zeros(m * nn, dtype=torch.float64, device="cuda")
    for di in (0, 1):
        for dj in (0, 1):
            w = (x - i if di else 1 - x + i) * (y - j if dj else 1 - y + j)
            want.index_add_(0, ((j + dj) * m + i + di).long(), w)
    want *= s.charge * parts.np2c / (grid.dx * grid.dy)
    assert (grid.rho.double() - want).abs().max() <= 1e-5 * want.abs().max()
    grid.E.copy_(torch.randn(2, m * nn, generator=g, device="cuda") * 1e3)
    v = [a.clone() for a in (s.vx, s.vy)]
    _lib.call("pic_update_V", _lib.ptr(s.x), _lib.ptr(s.y), _lib.ptr(v[0]), _lib.ptr(v[1]), s.n, _lib.ptr(grid.E[0]),
              _lib.ptr(grid.E[1]), m, nn, float(s.charge / s.mass * 1e-11), _lib.stream_ptr())
    parts.update_V(grid, 1e-11)
    assert grid._pairs is not None
    for a, b in zip(v, (s.vx, s.vy)):
        assert torch.equal(a.view(torch.int32), b.view(torch.int32))
