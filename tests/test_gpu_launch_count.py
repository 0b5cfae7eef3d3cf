"""pic_sim_kernel_launches against the kernels the profiler sees, for every way a step's
field solve runs: cycles in line that the solve needs and that it does not, the cooperative
launch after them, the loop node, captured steps and steps launched one by one, ensembles."""
import numpy as np
import pytest
import torch
from torch.profiler import ProfilerActivity, profile

from pic_b200 import Consts
from pic_b200.ensemble import Ensemble
from pic_b200.simulation import PICSimulation

pytestmark = pytest.mark.gpu
DX, N = 1e-4, 20_000


def make(nx, ny, tol, min_cycles=2, rz=False, use_graph=True, sort_interval=0, mg_launch="graph"):
    mask = np.zeros((ny, nx), np.uint8)
    mask[-1] = mask[:, 0] = mask[:, -1] = 1
    if not rz:
        mask[0] = 1
    sp = [dict(name=k, charge=q, mass=m, np2c=1e4, capacity=N)
          for k, q, m in (("e", -Consts.qe, Consts.me), ("i", Consts.qe, 40 * Consts.mp))]
    sim = PICSimulation(nx, ny, DX, DX, 1e-12, sp, mask, tol=tol, use_graph=use_graph, min_cycles=min_cycles,
                        max_cycles=11, sort_interval=sort_interval, geometry="rz" if rz else "cartesian",
                        mg_launch=mg_launch)
    rng = np.random.default_rng(nx)
    for s in (0, 1):
        sim.load(s, rng.uniform(1, nx - 2, N), rng.uniform(1, ny - 2, N), *[rng.normal(0, 1e5, N) for _ in range(3)])
    sim.init()
    return sim


def kernels(run):
    torch.cuda.synchronize()
    with profile(activities=[ProfilerActivity.CUDA], acc_events=True) as p:
        run()
        torch.cuda.synchronize()
    return sum(e.device_type == torch.autograd.DeviceType.CUDA and "mem" not in e.name.lower() for e in p.events())


@pytest.mark.parametrize("use_graph", [True, False])
@pytest.mark.parametrize("case", [dict(tol=1e-6), dict(tol=1e-8), dict(tol=1e-300), dict(tol=1e-8, min_cycles=0),
                                  dict(tol=1e-8, rz=True), dict(tol=1e-8, sort_interval=10),
                                  dict(tol=1e-8, nx=705, ny=641), dict(tol=1e-300, nx=705, ny=641),
                                  dict(tol=1e-8, nx=129, ny=129, mg_launch="dst")])
def test_launches_of_a_simulation(case, use_graph):
    case = dict(dict(nx=129, ny=97), **case)
    sim = make(use_graph=use_graph, **case)
    sim.step(12)
    before = sim.kernel_launches()
    seen = kernels(lambda: sim.step(20))
    assert sim.kernel_launches() - before == seen
    sim.close()


def test_launches_of_an_ensemble():
    sims = [make(129, 97, 1e-8), make(65, 65, 1e-300), make(129, 129, 1e-6, min_cycles=0)]
    for sim in sims:
        sim.step(2)
    ens = Ensemble(sims)
    ens.step(3)
    before = sum(s.kernel_launches() for s in sims)
    seen = kernels(lambda: ens.step(10))
    # what the graph adds for the whole ensemble is counted with no member
    counted = sum(s.kernel_launches() for s in sims) - before
    assert counted <= seen <= counted + 2 * 10, (counted, seen)
