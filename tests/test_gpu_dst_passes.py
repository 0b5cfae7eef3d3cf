"""The sine-transform solve at every FFT length (8 to 4096 points: one to four
radix-8 passes, the first of radix 2, 4 or 8) against the same solve by torch's FP64
FFT of the odd extension, on square and rectangular grids, odd row counts (the last
block holds one row), nonzero edges.

Tolerance: both are FP64 transforms of a few thousand points; 1e-12 of max|phi|.
"""
import math

import numpy as np
import pytest
import torch

from pic_b200.multigrid import MultigridSolver

HX, HY = 1e-3, 1.7e-3


def dst(a):
    z = torch.zeros_like(a[..., :1])
    return -0.5 * torch.fft.fft(torch.cat([z, a, z, -a.flip(-1)], -1)).imag[..., 1:a.shape[-1] + 1]


def lam(m, h):
    k = torch.arange(1, m - 1, dtype=torch.float64)
    return 4.0 / (h * h) * torch.sin(math.pi * k / (2.0 * (m - 1))) ** 2


@pytest.mark.gpu
@pytest.mark.parametrize("nx,ny", [(5, 5), (9, 5), (5, 17), (17, 9), (33, 33), (65, 17), (33, 129), (129, 257),
                                   (257, 65), (513, 513), (1025, 257), (513, 1025), (2049, 513), (513, 2049)])
def test_against_torch_fft(nx, ny):
    rng = np.random.default_rng(nx * 4096 + ny)
    mask = np.ones((ny, nx), np.uint8)
    mask[1:-1, 1:-1] = 0
    phi = torch.as_tensor(np.where(mask, rng.uniform(-40, 40, (ny, nx)), 0.0))
    f = torch.as_tensor(np.where(mask, 0.0, rng.normal(0, 1e6, (ny, nx))))
    b = f[1:-1, 1:-1].clone()
    b[:, 0] -= phi[1:-1, 0] / HX**2
    b[:, -1] -= phi[1:-1, -1] / HX**2
    b[0] -= phi[0, 1:-1] / HY**2
    b[-1] -= phi[-1, 1:-1] / HY**2
    u = dst(dst(b).T).T / -(lam(nx, HX)[None] + lam(ny, HY)[:, None])
    want = phi.clone()
    want[1:-1, 1:-1] = dst(dst(u).T).T * (4.0 / ((nx - 1) * (ny - 1)))
    mg = MultigridSolver(mask.reshape(-1), nx, ny, HX, hy=HY, launch="dst")
    assert mg.effective_launch() == "dst"
    got, _ = mg.solve(phi.reshape(-1).cuda(), f.reshape(-1).cuda(), tol=1e-9)
    got = got.cpu().reshape(ny, nx)
    assert torch.equal(got[torch.as_tensor(mask).bool()], phi[torch.as_tensor(mask).bool()])
    assert float((got - want).abs().max()) <= 1e-12 * float(want.abs().max())
