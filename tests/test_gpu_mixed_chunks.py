"""Chunks of every kind beside each other -- zeros, smooth, dense, incompressible
-- in launches with several chunks per CTA: what a CTA carries from one chunk to
the next (payloads waiting for their offset, buffers that change places) in every
order.  All operations, single and batched, streams and floats against the oracle."""
import numpy as np
import pytest
import torch

from oracle import oracle as O

pytestmark = pytest.mark.gpu

CW = 4096
OPS = ("store", "init_send", "resi_send", "store_decode", "init_recv", "resi_recv")
STORE, SRC, DST = 2e-4, 2e-3, 4e-4


@pytest.fixture(scope="module")
def codec(cuda_device):
    from cortado_b200.ops import Codec
    c = Codec(0)
    for op in OPS:
        c.set_launch_ctas(op, 1)
    yield c
    c.close()


def field(kinds, seed, tail):
    """One chunk per letter: zero, smooth, dense, random bits; then `tail` words of the last kind."""
    rng = np.random.Generator(np.random.PCG64(seed))
    out = []
    for i, k in enumerate(kinds):
        n = CW if i + 1 < len(kinds) or not tail else tail
        if k == "z":
            out.append(np.zeros(n, np.float32))
        elif k == "s":
            out.append((np.sin(np.arange(n) / 40.0) + rng.normal(0, 1e-3, n)).astype(np.float32))
        elif k == "d":
            out.append(rng.uniform(-2000, 2000, n).astype(np.float32))
        else:
            out.append(rng.integers(0, 1 << 32, n, dtype=np.uint32).view(np.float32))
    return np.concatenate(out)


def pattern(name, chunks):
    if name == "mixed":
        rng = np.random.Generator(np.random.PCG64(chunks))
        return "".join(rng.choice(list("zsdr"), chunks))
    return (name * chunks)[:chunks]


@pytest.mark.parametrize("name,tail", [("r", 0), ("zr", 17), ("zzzzzr", 0), ("d", 300), ("rd", 0), ("sr", 4095),
                                       ("z" * 70 + "r", 1), ("mixed", 2047), ("mixed", 0)])
def test_long_queues_match_oracle(codec, name, tail):
    from cortado_b200.ops import max_stream_bytes
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    # one field for the single calls; for the batched ones fields of uneven lengths
    lens = [5 * sms + 3, 2 * sms + 1, 1, 2 * sms]
    xs = [field(pattern(name, n), 10 * i + n, tail) for i, n in enumerate(lens)]
    dev = "cuda"
    state = []
    for x in xs:
        stor = O.store_encode(x, STORE)
        init, resi = O.init_send(stor, SRC), O.resi_send(stor, SRC, DST)
        rec = O.init_recv(init)
        state.append(dict(x=x, store=stor, init_send=init, resi_send=resi, init_recv=rec, store_decode=O.store_decode(stor),
                          resi_recv=O.resi_recv(rec, resi), n=4 * x.size, cap=max_stream_bytes(4 * x.size)))

    def up(b):
        return torch.from_numpy(np.frombuffer(bytes(b), np.uint8).copy()).to(dev)

    for s in state:
        s["g"] = {k: up(s[k]) for k in ("store", "init_send", "resi_send")}
        s["xg"] = torch.from_numpy(s["x"].copy()).to(dev)
        s["size"] = torch.zeros(1, dtype=torch.int64, device=dev)
        s["out"] = torch.zeros(s["cap"], dtype=torch.uint8, device=dev)
        s["f"] = torch.zeros(s["x"].size, device=dev)
        s["recg"] = torch.from_numpy(s["init_recv"].copy()).to(dev)

    def same_floats(t, want):
        return np.array_equal(t.cpu().numpy().view(np.uint32), np.asarray(want).view(np.uint32))

    def items(op, group):
        out = []
        for s in group:
            i = {"out_size": s["size"], "n_bytes": s["n"], "out": s["out"]}
            if op == "store":
                i.update({"in": s["xg"], "eb1": STORE})
            elif op.startswith("init_send"):
                i.update({"in": s["g"]["store"], "eb1": SRC})
            elif op.startswith("resi_send"):
                i.update({"in": s["g"]["store"], "eb1": SRC, "eb2": DST})
            else:
                i.update({"in": s["g"][{"store_decode": "store", "init_recv": "init_send", "resi_recv": "resi_send"}[op]],
                          "out": s["f"]})
            if op.endswith("_apply"):
                i["src"] = s["f"]
            if op == "resi_recv":
                i["src"] = s["recg"]
            out.append(i)
        return out

    def single(op, s):
        g, st = s["g"], s
        if op == "store":
            codec.server_encode(st["xg"], st["n"], st["out"], st["size"], STORE)
        elif op == "init_send":
            codec.s2c_encode(g["store"], st["out"], st["size"], SRC, st["n"])
        elif op == "resi_send":
            codec.residual_encode(g["store"], st["out"], st["size"], SRC, DST, st["n"])
        elif op == "init_send_apply":
            codec.s2c_encode_apply(g["store"], st["out"], st["size"], SRC, st["n"], st["f"])
        elif op == "resi_send_apply":
            codec.residual_encode_apply(g["store"], st["out"], st["size"], SRC, DST, st["n"], st["f"])
        elif op == "store_decode":
            codec.server_decode(g["store"], st["f"], st["size"])
        elif op == "init_recv":
            codec.client_decode(g["init_send"], st["f"], st["size"])
        else:
            codec.residual_apply(st["recg"], st["n"], g["resi_send"], st["f"], st["size"])

    for op in OPS + ("init_send_apply", "resi_send_apply"):
        for group in (state[:1], state):
            for s in group:
                s["out"].fill_(0xAA)
                s["f"].fill_(7.0)
                if op == "resi_send_apply":
                    s["f"].copy_(s["recg"])
            if len(group) == 1:
                single(op, group[0])
            else:
                codec.batch(op, items(op, group))
            codec.sync()
            for i, s in enumerate(group):
                base = op.removesuffix("_apply")
                if base in ("store", "init_send", "resi_send"):
                    got = bytes(s["out"][: int(s["size"].item())].cpu().numpy())
                    assert got == bytes(s[base]), (op, len(group), i)
                if op in ("store_decode", "init_recv", "resi_recv"):
                    assert same_floats(s["f"], s[op]), (op, len(group), i)
                elif op.endswith("_apply"):
                    assert same_floats(s["f"], s[{"init_send_apply": "init_recv", "resi_send_apply": "resi_recv"}[op]]), (op, len(group), i)
