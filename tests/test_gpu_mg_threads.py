"""Simulations stepped at the same time from threads and streams of their own, each step's
field solve ending in a cooperative launch whose blocks wait for one another: all of a
launch's blocks run at once whatever the other launches hold, so no barrier gives up.

Oracle: the same simulations stepped alone; cycles and residual as there.  Tolerance: the
residual is far below FP64's floor of the solve (see test_gpu_mg_rest)."""
import threading

import pytest
import torch

from test_gpu_mg_rest import CYCLES, make

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shapes", [[(513, 385)] * 3, [(129, 97), (513, 385), (65, 65), (257, 257)]])
def test_simulations_at_the_same_time(shapes):
    sims = [make(nx, ny, False)[0] for nx, ny in shapes]
    streams = [torch.cuda.Stream() for _ in sims]
    failed = []

    def run(sim, stream):
        try:
            with torch.cuda.stream(stream):
                for _ in range(10):
                    sim.step(5)
                sim.sync()
                c = sim.counters()
            assert c["last_cycles"] == CYCLES and c["last_rel_res"] < 1e-9
        except Exception as e:  # reported by the test's own thread
            failed.append(e)

    torch.cuda.synchronize()
    threads = [threading.Thread(target=run, args=a) for a in zip(sims, streams)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failed, failed
    for sim in sims:
        sim.close()
