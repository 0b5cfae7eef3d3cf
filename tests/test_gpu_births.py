"""MccOperator's birth arrays, taken and in place: each contiguous and aligned as a tensor
of its own (512 bytes, torch's allocations), whatever their number."""
import pytest
import torch

from pic_b200 import Consts, workloads
from pic_b200.MCC import MccOperator

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("capacity", [1, 127, 1001, 4096])
@pytest.mark.parametrize("count", [0, 1, 7, 126, 1001])
def test_birth_arrays_are_aligned(capacity, count):
    w = workloads.scaled(workloads.MCC, n=1000, nodes=65)
    op = MccOperator(workloads.mcc_tables(w), [Consts.me, workloads.ION_MASS], w.dt, birth_capacity=capacity)
    arrays = (op.bspecies, op.bx, op.by, op.bvx, op.bvy, op.bvz)
    for k, a in enumerate(arrays):
        a.copy_(torch.arange(capacity) + 10_000 * k)
    want = [a.cpu().clone() for a in arrays]
    op.bcount.fill_(count)
    taken = op.take_births()
    k = min(count, capacity)
    for a, b, w_ in zip(taken, arrays, want):
        assert a.is_contiguous() and a.dtype == b.dtype and torch.equal(a.cpu(), w_[:k])
        assert a.data_ptr() % 512 == 0 and b.data_ptr() % 512 == 0
    assert int(op.bcount) == 0
