"""The device bound check (MAXABS rules) on aligned arrays (16-byte loads) and
on arrays that start at an odd float (4-byte loads), at sizes around the ends
of a vector and of a pass: the first violating index, NaN and infinity
included, as the oracle reports it."""
import numpy as np
import pytest
import torch

from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def codec(cuda_device):
    from cortado_b200.ops import Codec
    c = Codec(0)
    yield c
    c.close()


@pytest.mark.parametrize("offset", [0, 1])
@pytest.mark.parametrize("words", [1, 3, 4, 5, 1023, 1024 * 148 * 8 + 7, 1 << 21])
def test_first_violation_matches_oracle(codec, words, offset):
    rng = np.random.Generator(np.random.PCG64(words + offset))
    x = rng.standard_normal(words).astype(np.float32)
    x[rng.integers(0, words, 3)] = np.inf
    good = (x + rng.uniform(-0.9e-3, 0.9e-3, words)).astype(np.float32)
    xg = torch.zeros(words + offset, device="cuda")[offset:]
    yg = torch.zeros(words + offset, device="cuda")[offset:]
    xg.copy_(torch.from_numpy(x))
    for bad in ([], [words - 1], [0, words - 1], list(rng.integers(0, words, 4))):
        y = good.copy()
        for n, i in enumerate(bad):
            y[i] = np.nan if n % 2 else x[i] + 1.0 if np.isfinite(x[i]) else 0.0
        yg.copy_(torch.from_numpy(y))
        first = codec.verify_bound(xg, yg, 1e-3)
        codec.sync()
        assert int(first.item()) == O.maxabs(y, x, 1e-3)
