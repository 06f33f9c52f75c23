"""The batch's sweeps at the edges of how their constants travel (16 and 128 instances as
kernel parameters, more in memory): an instance advances bit for bit as in a batch of its own."""
import numpy as np
import pytest

from sphinxsys_gb300 import cases
from sphinxsys_gb300.batch import BatchDamBreak

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim,count", [(2, 16), (2, 17), (2, 128), (2, 129), (3, 17)])
def test_instance_does_not_depend_on_the_batch(dim, count):
    inst = [c for c in cases.batch_instances(4 * count, seed=5, n_min=200, n_max=700) if c.dim == dim][:count]
    assert len(inst) == count
    many = BatchDamBreak(inst)
    for _ in range(2):
        many.advection_step()
    for q in (0, count // 2, count - 1):
        one = BatchDamBreak([inst[q]])
        for _ in range(2):
            one.advection_step()
        for a, b in zip(many.download(q), one.download(0)):
            assert np.array_equal(a, b), q
