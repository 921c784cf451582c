"""A batch whose instances are large enough for the two-pass kernels by node class (more than 7 Mi nodes), on the chain form, where
the step counts from a device counter: against each instance alone, bit for bit, probes in and outside the CPML among the results."""
import pytest

from conftest import bitwise_equal
from test_gpu_batch_sweep import drive
from test_gpu_sweep import case

pytestmark = pytest.mark.gpu


def test_chains_by_class(gpu_lib):
    import torch
    scs = [case((200, 196, 192), (6,) * 6, 3), case((40, 36, 34), (4,) * 6, 4)]
    calls, alone = (3, 34), (1, 2)
    want = drive(scs, [2, 1], calls, alone, None)
    got = drive(scs, [1, 1], calls, alone, (-1, 256))
    for (p, s), (q, t) in zip(got, want):
        assert bitwise_equal(p, q)
        assert torch.equal(s, t)
