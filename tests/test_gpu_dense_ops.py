"""The operators by 16-byte accesses and the collision operator's block split.

* pic_deposit_cells + pic_cells_density against the exact sum of the FP32
  contributions (the tolerance of the plain deposit: 2e-6 of the sum of their
  magnitudes), with particles on every edge and corner, dead slots, two signs.
* pic_field_pairs + pic_update_V_pairs against pic_update_V, bit for bit.
* Grid2D.update_density and Particles2D.update_V on both sides of the rule that
  picks them.
* pic_mcc_apply's candidates and per-process counts against the oracle's replay
  at slot counts around its blocks' 128 segments of 256, and with nearly every
  slot a candidate.
"""
import numpy as np
import pytest
import torch

from oracle import oracle as O
from pic_b200 import Consts, Grid, MCC, _lib, workloads
from pic_b200.Grid import Grid2D
from pic_b200.Particles import Particles2D

pytestmark = pytest.mark.gpu
DEV = "cuda"


def particles(rng, n, m, nn):
    x = rng.uniform(0, m - 1, n).astype(np.float32)
    y = rng.uniform(0, nn - 1, n).astype(np.float32)
    k = min(n, 4)
    x[:k] = np.array([0.0, m - 1, m - 1, 0.0], np.float32)[:k]
    y[:k] = np.array([0.0, nn - 1, 0.0, nn - 1], np.float32)[:k]
    if n > 64:
        x[4:20], y[20:36] = m - 1, nn - 1
        x[40:44] = np.nan
    return x, y


def dev(a):
    return torch.as_tensor(np.ascontiguousarray(a), device=DEV)


@pytest.mark.parametrize("m,nn,n", [(2, 2, 40), (17, 13, 1), (17, 13, 3000), (129, 65, 50_000), (130, 257, 300_001)])
def test_dense_deposit_and_gather(m, nn, n):
    rng = np.random.default_rng(m * n)
    st = _lib.stream_ptr()
    cells = torch.zeros((m * nn, 4), device=DEV)
    rho = torch.full((m * nn,), 7.0, device=DEV)
    exact, absum = np.zeros(m * nn), np.zeros(m * nn)
    loads = [particles(rng, n, m, nn) for _ in range(2)]
    for (x, y), scale in zip(loads, (np.float32(-3.7e-5), np.float32(2.9e-5))):
        X, Y = dev(x), dev(y)
        _lib.call("pic_deposit_cells", _lib.ptr(X), _lib.ptr(Y), n, float(scale), _lib.ptr(cells), m, nn, st)
        live = ~np.isnan(x)
        O.deposit_f32(x[live], y[live], scale, m, nn, exact, absum)
    _lib.call("pic_cells_density", _lib.ptr(cells), _lib.ptr(rho), m, nn, st)
    got = rho.cpu().numpy()
    assert np.all(np.abs(got - exact) <= 2e-6 * absum + 1e-30)
    E = dev(rng.normal(0, 1e3, (2, m * nn)).astype(np.float32))
    pairs = torch.empty((m * nn, 4), device=DEV)
    _lib.call("pic_field_pairs", _lib.ptr(E[0]), _lib.ptr(E[1]), _lib.ptr(pairs), m, nn, st)
    x, y = (dev(a) for a in loads[0])
    v = rng.normal(0, 1e5, (2, n)).astype(np.float32)
    a, b = dev(v[0]), dev(v[1])
    c, d = dev(v[0]), dev(v[1])
    _lib.call("pic_update_V", _lib.ptr(x), _lib.ptr(y), _lib.ptr(a), _lib.ptr(b), n, _lib.ptr(E[0]), _lib.ptr(E[1]), m,
              nn, 1.7, st)
    _lib.call("pic_update_V_pairs", _lib.ptr(x), _lib.ptr(y), _lib.ptr(c), _lib.ptr(d), n, _lib.ptr(pairs), m, nn, 1.7,
              st)
    assert torch.equal(a.view(torch.int32), c.view(torch.int32)) and torch.equal(b.view(torch.int32), d.view(torch.int32))


@pytest.mark.parametrize("cylindrical", [False, True])
def test_classes_give_the_same_on_both_sides_of_the_rule(cylindrical, monkeypatch):
    m, nn, n = 65, 33, 20_000
    out = []
    for dense in (False, True):
        monkeypatch.setattr(Grid, "DENSE_PARTICLES", 0 if dense else 1 << 30)
        grid = Grid2D(m, nn, 1e-4 * (m - 1), 1e-4 * (nn - 1), cylindrical=cylindrical)
        parts = Particles2D(n, cylindrical=cylindrical)
        parts.grid, parts.np2c = grid, 1e4
        for k, (name, mass, q) in enumerate((("e", Consts.me, -Consts.qe), ("i", workloads.ION_MASS, Consts.qe))):
            parts.add_species(name, mass, q, k)
            rng = np.random.default_rng(k)
            parts.load_species_arrays(k + 1, rng.uniform(0, grid.X, n), rng.uniform(0, grid.Y, n),
                                      rng.normal(0, 1e5, n), rng.normal(0, 1e5, n))
        grid.E.copy_(dev(np.random.default_rng(3).normal(0, 1e3, (2, m * nn)).astype(np.float32)))
        grid.update_density(parts)
        parts.update_V(grid, 1e-11)
        assert (grid._cells is not None) == dense and (grid._pairs is not None) == dense
        out.append((grid.rho.cpu().numpy(), [a.cpu().numpy() for s in parts.species for a in (s.vx, s.vy)]))
    scale = np.abs(out[0][0]).max()
    assert np.abs(out[0][0] - out[1][0]).max() <= 1e-5 * scale  # two species' sums of either sign nearly cancel
    for a, b in zip(out[0][1], out[1][1]):
        np.testing.assert_array_equal(a.view(np.uint32), b.view(np.uint32))


@pytest.mark.parametrize("n,density", [(1, 1e21), (255, 1e25), (32_768, 1e24), (32_769, 1e21), (100_003, 1e23)])
def test_mcc_counts_against_the_oracle(n, density):
    w = workloads.scaled(workloads.MCC, n=n, nodes=65, Te=20.0, gas_density=density)
    rng = np.random.Generator(np.random.Philox(n))
    arrays = list(workloads.species_arrays(w, "e", rng))
    if n > 300:
        arrays[0][100:110] = np.nan
    tables = workloads.mcc_tables(w)
    op = MCC.MccOperator(tables, [Consts.me, workloads.ION_MASS], w.dt, birth_capacity=1 << 18, seed=9)
    nu, p, inv = op.query(0)
    procs = tables.species[0]
    S, keep = O.mcc_species(tables.energy, [q[2] for q in procs], [q[0] for q in procs], [q[1] for q in procs],
                            tables.gas_density, Consts.me, tables.gas_mass, tables.gas_temperature, nu, inv, 0)
    d = [dev(a) for a in arrays]
    op.apply(0, *d, n, step=3)
    ctr = op.counters.cpu().numpy()
    cand = np.flatnonzero(O.mcc_candidates(S, n, 3, 9) & ~np.isnan(arrays[0]))
    assert ctr[16] == len(cand)
    counts = np.zeros(4, np.int64)
    moved = np.zeros(n, bool)
    for i in cand:
        proc, _, _ = O.mcc_collide(S, int(i), 3, 9, [a[i] for a in arrays[2:]])
        if proc >= 0:
            counts[proc] += 1
            moved[i] = True
    np.testing.assert_array_equal(ctr[:4], counts)
    for a, b in zip(arrays[2:], d[2:]):
        assert (a.view(np.uint32) == b.cpu().numpy().view(np.uint32))[~moved].all()
    births = op.take_births()
    assert births[0].numel() == 2 * ctr[2] and ctr[20] == 0
    assert int(op.bcount.item()) == 0 and births[0].dtype == torch.int32
