"""Batched receives in which items with unusable stream headers (wrong size,
corrupt exponent, a stream too short for its size table) lie between usable
ones, with many more chunks than CTAs, so that a CTA meets several unusable
chunks in a row and then a usable one.  The error is reported, nothing of an
unusable item is written, and every usable item's floats are bit-identical to
the oracle's.  Items stay below 256 chunks: their payload offsets never wait
for another CTA, whose failure would end the wait."""
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


def _spoil(stream, how):
    s = np.frombuffer(stream, np.uint8).copy()
    if how == 0:
        s[:8].view(np.int64)[0] += 4  # not the size that the caller gives
    elif how == 1:
        s[8:12].view(np.int32)[0] = 0  # no exponent
    else:
        s = s[:16].copy()  # a header without its size table
    return s


@pytest.mark.parametrize("op", ["store_decode", "init_recv", "resi_recv"])
def test_unusable_items_leave_the_others_alone(codec, op):
    from cortado_b200._native import CortadoError
    rng = np.random.Generator(np.random.PCG64(23))
    items = []  # (stream, client, floats expected or None, words)
    for i in range(240):
        words = int(rng.integers(1, 6)) * CW - int(rng.integers(0, 2)) * int(rng.integers(0, CW))
        x = (rng.uniform(-1, 1, words) * 1e-4 * 2.0 ** rng.integers(0, 20)).astype(np.float32)
        stor = O.store_encode(x, 1e-4, 1)
        init = O.init_send(stor, 1e-3, 1)
        client = O.init_recv(init, 1)
        resi = O.resi_send(stor, 1e-3, 1e-4, 1)
        stream, floats = {"store_decode": (stor, O.store_decode(stor, 1)), "init_recv": (init, client),
                          "resi_recv": (resi, O.resi_recv(client, resi, 1))}[op]
        bad = i < 4 or rng.random() < 0.6
        s = _spoil(stream, i % 3) if bad else np.frombuffer(stream, np.uint8).copy()
        items.append((torch.from_numpy(s).cuda(), torch.from_numpy(client.copy()).cuda(), None if bad else floats, words))
    sizes = torch.full((len(items),), -1, dtype=torch.int64, device="cuda")
    outs = [torch.full((w,), 7.0, device="cuda") for *_, w in items]
    codec.set_launch_ctas(op, 1)
    try:
        for _ in range(5):
            codec.batch(op, [{"in": s, "out": o, "out_size": sizes[i:], "n_bytes": 4 * w,
                              "src": c if op == "resi_recv" else None}
                             for i, ((s, c, _, w), o) in enumerate(zip(items, outs))])
            with pytest.raises(CortadoError) as e:
                codec.sync()
            assert e.value.name == "SIZE_MISMATCH"
            n = sizes.tolist()
            for i, (_, _, floats, words) in enumerate(items):
                got = outs[i].cpu().numpy()
                if floats is None:
                    assert n[i] == -1 and (got == 7.0).all(), i
                else:
                    assert n[i] == 4 * words and np.array_equal(got.view(np.uint32), floats.view(np.uint32)), i
                    outs[i].fill_(7.0)
            sizes.fill_(-1)
        codec.sync()  # reported once
    finally:
        codec.set_launch_ctas(op, 0)
