"""The kernels' per-chunk branches against the oracle: chunks from all-zero to
incompressible, with the numbers of non-zero words where the zero-byte
expansion and the compaction change their form, alone, in a partial last chunk
and followed by chunks of the other forms.  Streams are byte-identical and
decoded floats bit-identical."""
import numpy as np
import pytest
import torch

from oracle import oracle as O

pytestmark = pytest.mark.gpu

CW = 4096


@pytest.fixture(scope="module")
def codec(cuda_device):
    from cortado_b200.ops import Codec
    c = Codec(0)
    yield c
    c.close()


def field(spikes, words, seed):
    """`words` floats, zero but for `spikes` values per 4096 words (all of them
    noise when spikes is 4096)."""
    rng = np.random.Generator(np.random.PCG64(seed))
    x = np.zeros(words, np.float32)
    for c0 in range(0, words, CW):
        n = min(CW, words - c0)
        k = min(n, spikes)
        at = c0 + rng.choice(n, size=k, replace=False)
        x[at] = rng.uniform(-1, 1, k).astype(np.float32) * np.float32(10.0) ** rng.integers(-3, 4, k).astype(np.float32)
    return x


@pytest.mark.parametrize("words", [CW, 3 * CW, 2 * CW + 1, 2 * CW + 33, CW + 2047, 5 * CW - 1])
@pytest.mark.parametrize("spikes", [0, 1, 4, 12, 20, 40, 90, 200, 600, 4096])
def test_chunk_forms_match_oracle(codec, words, spikes):
    x = field(spikes, words, 1000 * spikes + words)
    if words == 5 * CW - 1:  # the other forms beside this one
        x[CW:2 * CW] = 0
        x[3 * CW:4 * CW] = field(4096, CW, words)
    xg = torch.from_numpy(x).cuda()

    def same(a, b):
        if isinstance(b, bytes):
            assert bytes(a.cpu().numpy()) == b
        else:
            assert np.array_equal(a.cpu().numpy().view(np.uint32), b.view(np.uint32))

    for store, src, dst in ((2e-6, 1e-2, 1e-4), (1e-3, 1e-1, 1e-3), (1e-3, 1e-4, 1e-2)):
        stor, ostor = codec.store(xg, store), O.store_encode(x, store)
        same(stor, ostor)
        same(codec.store_decode(stor), O.store_decode(ostor))
        init, oinit = codec.init_send(stor, src), O.init_send(ostor, src)
        same(init, oinit)
        rec, orec = codec.init_recv(init), O.init_recv(oinit)
        same(rec, orec)
        resi, oresi = codec.resi_send(stor, src, dst), O.resi_send(ostor, src, dst)
        same(resi, oresi)
        same(codec.resi_recv(rec, resi), O.resi_recv(orec, oresi))
