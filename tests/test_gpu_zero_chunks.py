"""Chunks whose words to encode are all zero skip the encode stage: zero fields,
fields whose stored bins vanish at the request or in the residual, and zeros
beside other chunks, with full and partial last chunks, single and batched.
Streams and the client's floats against the oracle."""
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


def field(kind, words):
    rng = np.random.Generator(np.random.PCG64(words))
    if kind == "zero":
        return np.zeros(words, np.float32)
    if kind == "signed":  # negative zeros and values below every bound
        x = np.full(words, -0.0, np.float32)
        x[::3] = 1e-9
        return x
    x = rng.uniform(-2e-3, 2e-3, words).astype(np.float32)  # bins at the stored bound, none at the request
    if kind == "mixed":
        x[(np.arange(words) // CW) % 2 == 0] = 0
        x[(np.arange(words) // CW) % 3 == 1] *= 1e6
    return x


@pytest.mark.parametrize("batched", [False, True])
@pytest.mark.parametrize("kind", ["zero", "signed", "vanishing", "mixed"])
@pytest.mark.parametrize("words", [1, 33, CW, 2 * CW + 1, 9 * CW + 2047])
def test_zero_chunks_match_oracle(codec, words, kind, batched):
    from cortado_b200.ops import max_stream_bytes
    x = field(kind, words)
    store, src, dst = 1e-4, 1e-1, 1e-1 if kind == "vanishing" else 1e-2
    stor = O.store_encode(x, store)
    init, resi = O.init_send(stor, src), O.resi_send(stor, src, dst)
    rec = O.init_recv(init)
    final = O.resi_recv(rec, resi)
    n, cap = 4 * words, max_stream_bytes(4 * words)
    sg = torch.from_numpy(np.frombuffer(stor, np.uint8).copy()).cuda()
    xg = torch.from_numpy(x).cuda()
    size = torch.zeros(1, dtype=torch.int64, device="cuda")
    out = torch.zeros(cap, dtype=torch.uint8, device="cuda")
    client = torch.full((words,), 7.0, device="cuda")

    def item(inp, **kw):
        return [{"in": inp, "out": out, "out_size": size, "n_bytes": n, **kw}]

    calls = {"store": (lambda: codec.server_encode(xg, n, out, size, store), item(xg, eb1=store), stor, None),
             "init_send": (lambda: codec.s2c_encode(sg, out, size, src, n), item(sg, eb1=src), init, None),
             "resi_send": (lambda: codec.residual_encode(sg, out, size, src, dst, n), item(sg, eb1=src, eb2=dst), resi, None),
             "init_send_apply": (lambda: codec.s2c_encode_apply(sg, out, size, src, n, client),
                                 item(sg, eb1=src, src=client), init, rec),
             "resi_send_apply": (lambda: codec.residual_encode_apply(sg, out, size, src, dst, n, client),
                                 item(sg, eb1=src, eb2=dst, src=client), resi, final)}
    for op, (call, batch, want, floats) in calls.items():
        out.fill_(0xAA)
        if op == "resi_send_apply":
            client.copy_(torch.from_numpy(rec.copy()))
        codec.batch(op, batch) if batched else call()
        codec.sync()
        assert bytes(out[: int(size.item())].cpu().numpy()) == want, op
        if floats is not None:
            assert np.array_equal(client.cpu().numpy().view(np.uint32), floats.view(np.uint32)), op
