"""The autotuner's thread choice where a CTA has its SM alone: there is one launch shape, and so nothing to
choose."""
import numpy as np
import pytest

from conicxx_gb300 import BatchSolver, generators

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("contacts", [10, 42])
@pytest.mark.parametrize("precision", [0, 1])
def test_tuning_a_batch_with_an_sm_for_every_instance_keeps_its_bits(contacts, precision):
    """No more instances than SMs: every candidate runs the same 256-thread block, and one that differs in the
    order of its sums alone would be taken by the noise of its timing."""
    B = BatchSolver([generators.contact_qp(s, contacts=contacts) for s in range(6)], precision=precision, warm_start=0)
    before, shape = B.solve(), B.describe()
    for _ in range(3):
        report = B.autotune(trials=1)
        assert B.describe() == shape
        assert "-> 256 threads" in report
        for a, b in zip(before[:3], B.solve()[:3]):
            assert np.array_equal(a, b)
