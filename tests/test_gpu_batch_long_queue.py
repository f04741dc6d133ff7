"""Batches of many more chunks than CTAs, so that every CTA works through
several chunks and what it carries from one to the next is exercised: a pending
payload beside the next stored one (and the flush when both do not fit), the
store's alternating buffers, the client's floats behind the next payload.
Short items whose last chunk is stored raw (1 to 300 floats) lie between items
whose payloads span the range from empty to uncompressed.  Streams are
byte-identical and floats bit-identical to the oracle's, item by item."""
import numpy as np
import pytest
import torch

from oracle import oracle as O

pytestmark = pytest.mark.gpu

CW = 4096
TAILS = (1, 5, 17, 33, 300)
ITEMS = 320  # 560 chunks or more: one CTA per SM takes three to four each


def _noise(rng, words, bits, eb):
    return (rng.uniform(-1, 1, words) * eb * 2.0**bits).astype(np.float32)


def make_items(seed=11):
    """(floats, store, request, source, destination bounds) per item."""
    rng = np.random.Generator(np.random.PCG64(seed))
    items = []
    for i in range(ITEMS):
        if i % 2:  # short: incompressible words, lossless at every bound but the source's
            words = TAILS[i // 2 % len(TAILS)] + (CW if i % 6 == 1 else 0)
            bits = rng.integers(0, 2**23, words, dtype=np.uint32) | (rng.integers(100, 140, words, dtype=np.uint32) << 23)
            bits |= rng.integers(0, 2, words, dtype=np.uint32) << 31
            items.append((bits.view(np.float32), 1e-30, 1e-30, 1e30, 1e-30))
        else:  # chunks of 0 to 26 significant bits a word
            eb = 1e-5
            parts = [_noise(rng, CW, int(b), eb) if b else np.zeros(CW, np.float32) for b in rng.integers(0, 27, 2)]
            if i % 8 == 0:
                parts.append(_noise(rng, int(rng.integers(1, CW)), int(rng.integers(1, 20)), eb))
            items.append((np.concatenate(parts), eb, eb * 8, eb * 8, eb))
    return items


def last_chunk_raw(stream, words):
    """Whether a stream's last chunk is stored uncompressed (size-table entry)."""
    chunks = -(-words // CW)
    entry = np.frombuffer(stream[16 + 2 * (chunks - 1):16 + 2 * chunks], np.uint16)[0]
    return int(entry) == 4 * (words - (chunks - 1) * CW)


def oracle_outputs(items):
    out = []
    for x, store, req, src, dst in items:
        stor = O.store_encode(x, store, 1)
        init = O.init_send(stor, req, 1)
        client = O.init_recv(O.init_send(stor, src, 1), 1)
        resi = O.resi_send(stor, src, dst, 1)
        out.append(dict(store=stor, store_decode=O.store_decode(stor, 1), init_send=init,
                        init_recv=O.init_recv(init, 1), resi_send=resi, client=client,
                        resi_recv=O.resi_recv(client, resi, 1)))
    return out


@pytest.fixture(scope="module")
def data():
    items = make_items()
    return items, oracle_outputs(items)


@pytest.fixture(scope="module")
def codec(cuda_device):
    from cortado_b200.ops import Codec
    c = Codec(0)
    yield c
    c.close()


def _dev(a):
    if isinstance(a, bytes):
        a = np.frombuffer(a, np.uint8)
    return torch.from_numpy(a.copy()).cuda()


@pytest.mark.parametrize("op", ["store", "store_decode", "init_send", "init_recv", "resi_send", "resi_recv",
                                "init_send_apply", "resi_send_apply"])
def test_long_queue_matches_oracle(codec, data, op):
    from cortado_b200.ops import max_stream_bytes
    items, want = data
    base = op.replace("_apply", "")
    source = {"store_decode": "store", "init_send": "store", "resi_send": "store", "init_recv": "init_send",
              "resi_recv": "resi_send"}
    for it, w in zip(items[1::2], want[1::2]):  # what the short items are there for
        assert last_chunk_raw(w["init_send"], it[0].size) and last_chunk_raw(w["resi_send"], it[0].size)
    sends = base in ("store", "init_send", "resi_send")
    ins = [_dev(x if op == "store" else w[source[base]]) for (x, *_), w in zip(items, want)]
    sizes = torch.zeros(len(items), dtype=torch.int64, device="cuda")
    outs = [torch.zeros(max_stream_bytes(4 * x.size) if sends else 4 * x.size, dtype=torch.uint8, device="cuda")
            for x, *_ in items]
    clients = [_dev(w["client"]) for w in want]
    batch = []
    for i, (x, store, req, src, dst) in enumerate(items):
        eb1 = {"store": store, "init_send": req, "resi_send": src}.get(base, 0.0)
        batch.append({"in": ins[i], "out": outs[i], "out_size": sizes[i:], "n_bytes": 4 * x.size, "eb1": eb1,
                      "eb2": dst, "src": clients[i] if base == "resi_recv" or op != base else None})
    codec.set_launch_ctas(base, 1)
    try:
        for _ in range(3):  # chunks are dealt out in another order each time
            for c, w in zip(clients, want):
                c.copy_(_dev(w["client"]))
            codec.batch(op, batch)
            codec.sync()
            n = sizes.tolist()
            for i, w in enumerate(want):
                ref = w[base] if isinstance(w[base], bytes) else w[base].tobytes()
                assert bytes(outs[i][:n[i]].cpu().numpy()) == ref, (op, i)
                if op != base:
                    got = clients[i].cpu().numpy().view(np.uint32)
                    assert np.array_equal(got, w["init_recv" if base == "init_send" else "resi_recv"].view(np.uint32)), (op, i)
    finally:
        codec.set_launch_ctas(base, 0)
