"""The multigrid's register tiles (pic_b200/csrc/mg_regtile.cuh) against whole-level
numpy phases in FP64.

One and three V-cycles of the FP64 solver, from a random potential, must give the
potential that the same cycle gives when every phase runs over the whole level:
red-black sweeps from zero, the residual and its full weighting, an exact solve of
the first level of at most 33^2 nodes, bilinear prolongation, sweeps.  Grids end
just before, on and after tile boundaries (cores of 54, 52, 56, 36 nodes and the
lower blocks' 22, 38, 20, 4 rows), rectangular ones among them, Cartesian and r-z,
with electrodes on odd lines, one to three sweeps each way, with one and with two
levels per launch.  The mixed solver's cycles are FP32: it must reach the same
potential to a residual tolerance, in the same number of cycles as the host loop.

Tolerance: FP64 rounding of the phases (a few hundred operations per node and
cycle, values of order max|phi|): 1e-12 of max|phi|.
"""
import numpy as np
import pytest
import scipy.sparse as sp
import scipy.sparse.linalg as spla
import torch

from pic_b200.multigrid import MultigridSolver

DX, DY, OMEGA = 1e-4, 1.3e-4, 1.15


def weights(ny, hx, hy, rz):
    """cx, and per row the weights of rows j+1 and j-1, the diagonal, the volume weight."""
    j = np.arange(ny, dtype=np.float64)
    cy = 1.0 / (hy * hy)
    if not rz:
        return 1.0 / (hx * hx), np.full(ny, cy), np.full(ny, cy), np.full(ny, 2.0 / (hx * hx) + 2 * cy), np.ones(ny)
    jj = np.maximum(j, 1)
    wn, ws = cy * (1 + 0.5 / jj), cy * (1 - 0.5 / jj)
    wn[0], ws[0] = 4 * cy, 0.0
    D = j.copy()
    D[0] = 0.125
    return 1.0 / (hx * hx), wn, ws, 2.0 / (hx * hx) + wn + ws, D


def neighbours(e, cx, wn, ws):
    p = np.pad(e, 1)
    return cx * (p[1:-1, :-2] + p[1:-1, 2:]) + wn[:, None] * p[2:, 1:-1] + ws[:, None] * p[:-2, 1:-1]


def sweeps(e, g, free, W, n):
    cx, wn, ws, diag, _ = W
    parity = np.add.outer(np.arange(e.shape[0]), np.arange(e.shape[1])) % 2
    for _ in range(n):
        for color in (0, 1):
            upd = (neighbours(e, cx, wn, ws) - g) / diag[:, None]
            e = np.where(free & (parity == color), e + OMEGA * (upd - e), e)
    return e


def restrict(r, rz):
    h = 0.5 * r[:, ::2]
    p = np.pad(r, ((0, 0), (1, 1)))
    h = h + 0.25 * (p[:, :-2:2] + p[:, 2::2])
    q = np.pad(h, ((1, 1), (0, 0)))
    v = 0.5 * h[::2] + 0.25 * (q[:-2:2] + q[2::2])
    if rz:
        J = np.arange(v.shape[0], dtype=np.float64)
        v = v * np.where(J == 0, 3.2, 0.5 / np.maximum(J, 1))[:, None]
    return v


def prolong(c):
    f = np.zeros((2 * c.shape[0] - 1, 2 * c.shape[1] - 1))
    f[::2, ::2] = c
    f[::2, 1::2] = 0.5 * (c[:, :-1] + c[:, 1:])
    f[1::2] = 0.5 * (f[:-2:2] + f[2::2])
    return f


def coarse_free(free, rz):
    """A coarse node is free unless its injected fine node is fixed, an internal
    fixed node lies in its 3 x 3 fine neighbourhood, or it is on an edge."""
    inner = ~free
    inner[-1] = inner[:, 0] = inner[:, -1] = False
    if not rz:
        inner[0] = False
    p = np.pad(inner, 1)
    near = np.zeros_like(inner)
    for dj in range(3):
        for di in range(3):
            near |= p[dj:dj + inner.shape[0], di:di + inner.shape[1]]
    return free[::2, ::2] & ~near[::2, ::2]


def exact(g, free, W):
    cx, wn, ws, diag, _ = W
    ny, nx = g.shape
    A = sp.diags(np.repeat(-diag, nx)).tolil()
    idx = np.arange(ny * nx).reshape(ny, nx)
    for j in range(ny):
        for i in range(nx):
            if free[j, i]:
                for jj, ii, w in ((j, i - 1, cx), (j, i + 1, cx), (j + 1, i, wn[j]), (j - 1, i, ws[j])):
                    if 0 <= jj < ny and free[jj, ii]:
                        A[idx[j, i], idx[jj, ii]] = w
    f = free.reshape(-1)
    e = np.zeros(ny * nx)
    e[f] = spla.spsolve(A.tocsr()[f][:, f].tocsc(), g.reshape(-1)[f])
    return e.reshape(ny, nx)


def vcycle(g, free, hx, hy, rz, pre, post):
    W = weights(g.shape[0], hx, hy, rz)
    if g.size <= 33 * 33:
        return exact(g, free, W)
    cx, wn, ws, diag, D = W
    e = sweeps(np.zeros_like(g), g, free, W, pre)
    r = np.where(free, D[:, None] * (g - (neighbours(e, cx, wn, ws) - diag[:, None] * e)), 0.0)
    cf = coarse_free(free, rz)
    c = vcycle(np.where(cf, restrict(r, rz), 0.0), cf, 2 * hx, 2 * hy, rz, pre, post)
    return sweeps(np.where(free, e + prolong(c), 0.0), g, free, W, post)


def problem(nx, ny, rz, electrode):
    rng = np.random.default_rng(nx * 1000 + ny)
    free = np.zeros((ny, nx), bool)
    free[0 if rz else 1:-1, 1:-1] = True
    if electrode:
        free[ny // 3:ny // 2, (nx // 4) | 1] = False
        free[(ny // 5) | 1, nx // 2:nx // 2 + 7] = False
    phi = np.where(free, 0.0, rng.uniform(-50.0, 50.0, (ny, nx)))
    f = np.where(free, rng.normal(0.0, 1e6, (ny, nx)), 0.0)
    return free, phi, f


GRIDS = [(49, 65), (57, 41), (97, 65), (105, 113), (161, 97), (225, 129), (257, 145), (321, 193)]


@pytest.mark.gpu
@pytest.mark.parametrize("sw", [(1, 1), (2, 2), (3, 3), (3, 1)])
@pytest.mark.parametrize("rz", [False, True])
@pytest.mark.parametrize("shape", GRIDS)
def test_cycles_against_whole_level_phases(shape, rz, sw):
    nx, ny = shape
    free, phi0, f = problem(nx, ny, rz, electrode=sw != (1, 1))
    W = weights(ny, DX, DY, rz)
    mg = MultigridSolver((~free).astype(np.uint8).reshape(-1), nx, ny, DX, omega=OMEGA, precision="fp64", hy=DY,
                         pre_sweeps=sw[0], post_sweeps=sw[1], geometry="rz" if rz else "cartesian")
    for cycles in (1, 3):
        want = phi0.copy()
        for _ in range(cycles):
            r = np.where(free, f - (neighbours(want, *W[:3]) - W[3][:, None] * want), 0.0)
            want = want + vcycle(r, free, DX, DY, rz, *sw)
        phi = torch.as_tensor(phi0.reshape(-1).copy(), device="cuda")
        phi, (n, rel) = mg.solve(phi, torch.as_tensor(f.reshape(-1), device="cuda"), tol=1e-300, max_cycles=cycles)
        assert n == cycles
        got = phi.cpu().numpy().reshape(ny, nx)
        np.testing.assert_allclose(got, want, rtol=0, atol=1e-12 * np.abs(want).max())
        # the residual kept from cycle to cycle, and its norm
        res = np.where(free, f - (neighbours(got, *W[:3]) - W[3][:, None] * got), 0.0)
        assert abs(rel / (np.linalg.norm(res) / np.linalg.norm(f)) - 1.0) < 1e-6


@pytest.mark.gpu
@pytest.mark.parametrize("max_cycles", [1, 2, 4, 5, 40])
@pytest.mark.parametrize("precision", ["mixed", "fp64"])
def test_cycles_launched_ahead_stop_where_the_host_loop_stops(precision, max_cycles):
    """Cycles in line before the loop node, skipped once the solve has ended: the same
    cycle count, residual and potential as the host-driven loop, from a poor guess, a
    good one and a converged one."""
    nx, ny = 129, 97
    free, phi0, f = problem(nx, ny, False, electrode=False)
    mask = (~free).astype(np.uint8).reshape(-1)
    F = torch.as_tensor(f.reshape(-1), device="cuda")
    graph = MultigridSolver(mask, nx, ny, DX, precision=precision, hy=DY)
    host = MultigridSolver(mask, nx, ny, DX, precision=precision, hy=DY, launch="host")
    guess = torch.as_tensor(phi0.reshape(-1).copy(), device="cuda")
    for tol in (1e-3, 1e-9):
        a, b = guess.clone(), guess.clone()
        for _ in range(3):  # the second and third start from the last solution
            _, (na, ra) = graph.solve(a, F, tol=tol, max_cycles=max_cycles)
            _, (nb, rb) = host.solve(b, F, tol=tol, max_cycles=max_cycles)
            assert na == nb and abs(ra - rb) <= 1e-6 * rb + 1e-14
            scale = float(b.abs().max())
            assert float((a - b).abs().max()) <= 1e-12 * scale


@pytest.mark.gpu
def test_changing_buffers_and_limits():
    """A solver given a new pair of buffers on each call, and the first pair again with
    other limits, solves each as a solver of its own would."""
    nx, ny = 129, 97
    free, phi0, f = problem(nx, ny, False, electrode=True)
    mask = (~free).astype(np.uint8).reshape(-1)
    shared = MultigridSolver(mask, nx, ny, DX, hy=DY)
    keep = []
    for k, tol in enumerate((1e-6, 1e-6, 1e-9, 1e-9, 1e-6)):
        F = torch.as_tensor((f * (k + 1)).reshape(-1).copy(), device="cuda")
        a = torch.as_tensor(phi0.reshape(-1).copy(), device="cuda")
        b = a.clone()
        keep += [F, a]  # no buffer is handed out twice
        _, (na, ra) = shared.solve(a, F, tol=tol)
        _, (nb, rb) = MultigridSolver(mask, nx, ny, DX, hy=DY).solve(b, F, tol=tol)
        assert na == nb and torch.equal(a, b)
    first = keep[1]
    first.copy_(torch.as_tensor(phi0.reshape(-1).copy()))
    b = first.clone()
    shared.solve(first, keep[0], tol=1e-10)
    MultigridSolver(mask, nx, ny, DX, hy=DY).solve(b, keep[0], tol=1e-10)
    assert torch.equal(first, b)


@pytest.mark.gpu
@pytest.mark.parametrize("sw", [1, 2, 3])
@pytest.mark.parametrize("rz", [False, True])
@pytest.mark.parametrize("precision", ["mixed", "fp64"])
@pytest.mark.parametrize("shape", [(49, 65), (129, 97), (321, 193), (609, 609), (641, 609)])
def test_cycles_after_the_launched_ones(shape, precision, rz, sw):
    """The cycles past those launched in line (one cooperative launch where a phase is one
    wave of tiles, up to 609 x 609 here, and no electrode is inside; else the loop node) end in
    the host loop's cycle, residual and potential, cut off by max_cycles and by the tolerance,
    from a poor guess and from a good one.  FP64: as above.  FP32 cycles: the same operations on corrections that
    are below 1e-2 of the potential by then, rounded at 6e-8: 1e-9 of it."""
    nx, ny = shape
    free, phi0, f = problem(nx, ny, rz, electrode=nx == 321)
    mask = (~free).astype(np.uint8).reshape(-1)
    F = torch.as_tensor(f.reshape(-1), device="cuda")
    o = dict(precision=precision, hy=DY, pre_sweeps=sw, post_sweeps=sw, geometry="rz" if rz else "cartesian")
    graph = MultigridSolver(mask, nx, ny, DX, **o)
    host = MultigridSolver(mask, nx, ny, DX, launch="host", **o)
    for tol, limit in ((1e-300, 10), (1e-3, 60), (1e-10, 60)):
        a = torch.as_tensor(phi0.reshape(-1).copy(), device="cuda")
        b = a.clone()
        for _ in range(2):
            _, (na, ra) = graph.solve(a, F, tol=tol, max_cycles=limit)
            _, (nb, rb) = host.solve(b, F, tol=tol, max_cycles=limit)
            assert na == nb and (tol > 1e-300 or na == limit)
            assert abs(ra - rb) <= (1e-3 if precision == "mixed" else 1e-6) * rb + 1e-11
            scale = float(b.abs().max())
            assert float((a - b).abs().max()) <= (1e-9 if precision == "mixed" else 1e-12) * scale


@pytest.mark.gpu
@pytest.mark.parametrize("sw", [1, 2, 3])
@pytest.mark.parametrize("rz", [False, True])
def test_cycles_of_more_than_one_wave_of_tiles(rz, sw):
    """Grids of more tiles than the GPU has SMs, where the residual up phase keeps the
    potential and the residual in shared memory: FP64 as above; one cycle in FP32 on the
    same whole-level phases, a hundred operations in a row rounded at 6e-8: 2e-5 of
    max|phi|."""
    nx, ny = 705, 641
    test_cycles_against_whole_level_phases((nx, ny), rz, (sw, sw))
    free, phi0, f = problem(nx, ny, rz, electrode=True)
    W = weights(ny, DX, DY, rz)
    mg = MultigridSolver((~free).astype(np.uint8).reshape(-1), nx, ny, DX, omega=OMEGA, precision="mixed", hy=DY,
                         pre_sweeps=sw, post_sweeps=sw, geometry="rz" if rz else "cartesian")
    r = np.where(free, f - (neighbours(phi0, *W[:3]) - W[3][:, None] * phi0), 0.0)
    want = phi0 + vcycle(r, free, DX, DY, rz, sw, sw)
    phi = torch.as_tensor(phi0.reshape(-1).copy(), device="cuda")
    mg.solve(phi, torch.as_tensor(f.reshape(-1), device="cuda"), tol=1e-300, max_cycles=1)
    np.testing.assert_allclose(phi.cpu().numpy().reshape(ny, nx), want, rtol=0, atol=2e-5 * np.abs(want).max())
