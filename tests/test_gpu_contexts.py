"""Contexts that are created and destroyed again and again, several alive at once,
each with its own scratch: streams of chunks that do not compress, which the
re-encoders keep there, stay right."""
import numpy as np
import pytest
import torch

from oracle import oracle as O

pytestmark = pytest.mark.gpu


def test_contexts_in_turn_and_side_by_side(cuda_device):
    from cortado_b200.ops import Codec
    rng = np.random.Generator(np.random.PCG64(3))
    xs = [rng.integers(0, 1 << 32, 60 * 4096 + 9, dtype=np.uint32).view(np.float32) for _ in range(6)]
    stored = [O.store_encode(x, 1e-3) for x in xs]
    want = [O.init_send(s, 1e-2) for s in stored]
    gpu = [torch.from_numpy(np.frombuffer(s, np.uint8).copy()).cuda() for s in stored]
    for alive in (1, 6, 2):
        codecs = [Codec(0) for _ in range(alive)]
        streams = [torch.cuda.Stream() for _ in range(alive)]
        outs = [torch.zeros(gpu[i].numel() + 65536, dtype=torch.uint8, device="cuda") for i in range(alive)]
        sizes = [torch.zeros(1, dtype=torch.int64, device="cuda") for _ in range(alive)]
        torch.cuda.synchronize()
        for i, c in enumerate(codecs):
            for _ in range(3):
                c.s2c_encode(gpu[i], outs[i], sizes[i], 1e-2, 4 * xs[i].size, stream=streams[i])
        for i, c in enumerate(codecs):
            c.sync(streams[i])
            assert bytes(outs[i][: int(sizes[i].item())].cpu().numpy()) == want[i]
        for c in codecs:
            c.close()
