"""The device bound check on arrays that start at an odd float: the first
violating index at the ends of the kernel's passes of eight loads per thread,
as the oracle reports it."""
import numpy as np
import pytest
import torch

from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("extra", [-1, 0, 1, 12345])
def test_first_violation_over_passes(cuda_device, extra):
    from cortado_b200.ops import Codec
    codec = Codec(0)
    stride = 8 * torch.cuda.get_device_properties(0).multi_processor_count * 256
    words = 16 * stride + extra
    x = np.random.Generator(np.random.PCG64(words)).standard_normal(words).astype(np.float32)
    xg = torch.zeros(words + 1, device="cuda")[1:]
    yg = torch.zeros(words + 1, device="cuda")[1:]
    xg.copy_(torch.from_numpy(x))
    last = words - 1
    # (the fourth: one thread's indices of the same pass, the later one listed first)
    for bad in ([], [last], [8 * stride, last], [7 * stride + 5, stride + 5], [8 * stride - 1, last]):
        y = x.copy()
        y[bad] = np.nan
        yg.copy_(torch.from_numpy(y))
        first = codec.verify_bound(xg, yg, 1e-3)
        codec.sync()
        assert int(first.item()) == O.maxabs(y, x, 1e-3) == (min(bad) if bad else -1)
    codec.close()
