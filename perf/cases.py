"""The calls that a user of this package times: what they do, on which data, and what they return.

Every case runs public entry points (``ops.Codec``, ``chain.ProgressiveChain``) on float32 fields that are resident
on the GPU, as a program that owns its buffers calls them.  A case is a dict:

* ``op``: what one pass does (``run`` below);
* ``words``: floats in the field (``rows`` x ``cols`` for the chain; ``fields``, ``least`` and ``most`` for a batch:
  that many fields, from ``least`` to ``most`` floats in a geometric progression, every size odd or even as it falls);
* ``kind``: the field's generator: ``sinusoid`` (8 waves plus noise), ``outliers`` (the same with 0.1% of the values
  at +-1e6), ``grf`` (Gaussian random field) or ``white``; a batch cycles through three of them;
* ``mode``: how the bounds are given: ``abs`` (absolute), ``noa`` (relative to the value range, which stays on the
  device) or ``host`` (relative, scaled on the host after the range has come back);
* ``store``, ``init``, ``dst``: the stored bound, the first request's and the refinement's.
"""
import math

import torch

from cortado_b200 import storage
from cortado_b200.chain import ProgressiveChain
from cortado_b200.ops import Codec, max_stream_bytes

CHAIN_STORE = (1e-1, 1e-3, 1e-5, 1e-7)
CHAIN_STEPS = (1e-1, 1e-2, 1e-3, 1e-4, 1e-5, 1e-6)
BATCH_STORE = (1e-1, 1e-2, 1e-3, 1e-4)
KINDS = ("sinusoid", "grf", "white")


def listed():
    big = 512 * 512 * 512
    return [
        # the smallest field of a collection through the whole exchange, six calls: launches and latency count
        dict(name="flow_small", op="flow", words=263167, kind="sinusoid", mode="noa", store=1e-4, init=1e-2, dst=1e-3),
        # a 128^3 field stored the way the command-line tool does it: range to the host, bound scaled there
        dict(name="store_128", op="store", words=128 * 128 * 128, kind="sinusoid", mode="host", store=1e-5),
        # a large field with outliers at a relative bound: nearly all bins are zero
        dict(name="store_large", op="store", words=big, kind="outliers", mode="noa", store=1e-4),
        # the same field at a tight absolute bound: dense chunks, some lossless words
        dict(name="store_dense", op="store", words=big, kind="outliers", mode="abs", store=1e-6),
        # reading a stored field back (an archive's decode), odd size
        dict(name="load_mid", op="load", words=60000001, kind="grf", mode="noa", store=1e-4),
        # a server answering a first request from a stored field
        dict(name="send_large", op="init_send", words=big, kind="outliers", mode="noa", store=1e-4, init=1e-2),
        # the client's side of a first request on dense data
        dict(name="recv_mid", op="init_recv", words=100000771, kind="sinusoid", mode="abs", store=1e-4, init=1e-3),
        # a server refining a client from 1e-3 to 1e-5 on dense data
        dict(name="resi_send_mid", op="resi_send", words=67109891, kind="outliers", mode="abs", store=1e-6, init=1e-3,
             dst=1e-5),
        # the client's side of the refinement
        dict(name="resi_recv_mid", op="resi_recv", words=90000001, kind="sinusoid", mode="noa", store=1e-4, init=1e-2,
             dst=1e-4),
        # an archive job: many fields of uneven sizes, each at four bounds, one launch
        dict(name="batch_store", op="batch_store", fields=12, least=262144, most=12582912, mode="host"),
        # a server's batches: every client of many fields opens its field, then refines it
        dict(name="batch_serve", op="batch_serve", fields=10, least=1048576, most=33554432, mode="host", store=1e-4,
             init=1e-2, dst=1e-3),
        # a progressive session captured once and replayed: first request and five refinements, each bound checked
        dict(name="chain", op="chain", rows=5000, cols=6001, kind="grf", mode="host"),
    ]


def draw(rng):
    def size(least, most):
        n = int(math.exp(rng.uniform(math.log(least), math.log(most))))
        return n - n % 4096 if n % 4096 < 512 else n  # a last chunk of a few floats is stored raw and has no 64-bit value

    ops = ("store", "store", "load", "init_send", "init_recv", "resi_send", "resi_recv", "flow", "step", "batch_store",
           "batch_serve", "chain")
    op = rng.choice(ops)
    case = dict(op=op, mode=rng.choice(("abs", "noa", "host")))
    if op == "chain":
        rows, cols = rng.randint(300, 5000), rng.randint(300, 6000)
        while 0 < rows * cols % 4096 < 512:
            cols += 1
        return dict(case, mode="host", kind="grf", rows=rows, cols=cols)
    if op == "batch_store":
        return dict(case, mode="host", fields=rng.randint(3, 12), least=size(65536, 262144), most=size(524288, 12582912))
    fine = rng.uniform(-5, -3)
    mid = rng.uniform(max(fine + 0.3, -4), -1.5)
    bounds = dict(store=10**fine, init=10**mid, dst=10 ** rng.uniform(fine + 0.05, mid - 0.1))
    if op == "batch_serve":
        return dict(case, mode="host", fields=rng.randint(3, 10), least=size(65536, 1048576), most=size(2097152, 33554432),
                    **bounds)
    case.update(words=size(65536, 60000000), kind=rng.choice(("sinusoid", "outliers", "grf", "white")), **bounds)
    if op in ("flow", "step"):
        case["mode"] = "noa"
    return case


# ------------------------------------------------------------------ fields
def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _sinusoid(words, g):
    side = 128 if words < 8388608 else 512
    rows = -(-words // (side * side))
    amp = torch.empty(8, device="cuda").uniform_(0.1, 1.0, generator=g)
    k = torch.empty(8, 3, device="cuda").uniform_(1.0, 16.0, generator=g) * (2 * math.pi)
    phi = torch.empty(8, device="cuda").uniform_(0.0, 2 * math.pi, generator=g)
    x, y, z = (torch.arange(n, device="cuda", dtype=torch.float32) / n for n in (rows, side, side))
    a = (x[:, None, None] * k[:, 0] + y[:, None] * k[:, 1] + phi).reshape(-1, 8)
    b = z[None, :] * k[:, 2, None]
    out = (torch.cos(a) * amp) @ torch.cos(b) - (torch.sin(a) * amp) @ torch.sin(b)
    out = out.reshape(-1)[:words].contiguous()
    return out.add_(torch.randn(words, device="cuda", generator=g), alpha=1e-3)


def _grf(shape, slope, g):
    spec = torch.fft.rfftn(torch.randn(shape, device="cuda", generator=g))
    freqs = [torch.fft.fftfreq(n, device="cuda") * n for n in shape[:-1]]
    freqs.append(torch.fft.rfftfreq(shape[-1], device="cuda") * shape[-1])
    k2 = torch.zeros(spec.shape, device="cuda")
    for axis, f in enumerate(freqs):
        k2 += (f**2).view([-1 if i == axis else 1 for i in range(len(shape))])
    zero = (0,) * len(shape)
    k2[zero] = 1.0
    spec *= k2.pow_(-slope / 4)
    spec[zero] = 0
    out = torch.fft.irfftn(spec, s=shape).reshape(-1)
    return out / out.std()


def _field(words, kind, seed):
    g = _generator(seed)
    if kind == "white":
        return torch.empty(words, device="cuda").uniform_(-1, 1, generator=g)
    if kind == "grf":
        side = 128 if words < 8388608 else 256
        return _grf((-(-words // (side * side)), side, side), 3.0, g)[:words].contiguous()
    x = _sinusoid(words, g)
    if kind == "outliers":
        at = torch.randint(0, words, (words // 1000,), device="cuda", generator=g)
        x[at] = 1e6
        x[at[: at.numel() // 2]] = -1e6
    return x


def _batch_sizes(case):
    n, lo, hi = case["fields"], case["least"], case["most"]
    sizes = (int(lo * (hi / lo) ** (i / (n - 1))) for i in range(n))
    return [s - s % 4096 if s % 4096 < 512 else s for s in sizes]


def _inputs(case, seed):
    if case["op"] == "chain":
        return [_grf((case["rows"], case["cols"]), 2.5, _generator(seed))]
    if "fields" in case:
        return [_field(n, KINDS[i % 3], seed * 1000 + i) for i, n in enumerate(_batch_sizes(case))]
    return [_field(case["words"], case["kind"], seed)]


def _scaled(case, x, bound):
    """The absolute bound, as the host computes it."""
    if case["mode"] == "abs":
        return float(storage.f32(bound))
    return float(storage.noa_scale(bound, storage.value_range(float(x.min()), float(x.max()))))


# ------------------------------------------------------------------ what a program holds before the call
def prepare(case, seed):
    op, xs = case["op"], _inputs(case, seed)
    codec = Codec()
    state = dict(case=case, codec=codec)
    if op == "chain":
        x = xs[0]
        codec.reserve(-(-x.numel() // 4096))
        chain = ProgressiveChain(codec, x, [_scaled(case, x, b) for b in CHAIN_STORE], _scaled(case, x, CHAIN_STEPS[0]),
                                 [_scaled(case, x, b) for b in CHAIN_STEPS[1:]])
        for s in chain.streams:
            s.zero_()
        chain.capture()
        return dict(state, chain=chain)
    if "fields" in case:
        per = len(BATCH_STORE) if op == "batch_store" else 2
        room = [-(-max_stream_bytes(4 * x.numel()) // 256) * 256 for x in xs for _ in range(per)]
        arena = torch.zeros(sum(room), dtype=torch.uint8, device="cuda")
        outs = list(arena.split(room))
        sizes = torch.zeros(len(outs), dtype=torch.int64, device="cuda")
        codec.reserve(per * sum(-(-x.numel() // 4096) for x in xs), len(outs))
        state.update(arena=arena, sizes=sizes)
        if op == "batch_store":
            items = [{"in": x, "out": outs[4 * i + j], "out_size": sizes[4 * i + j:], "n_bytes": 4 * x.numel(),
                      "eb1": _scaled(case, x, b)} for i, x in enumerate(xs) for j, b in enumerate(BATCH_STORE)]
            return dict(state, x=xs, items=items)
        clients = [torch.zeros_like(x) for x in xs]
        first, second = [], []
        for i, x in enumerate(xs):
            eb = [_scaled(case, x, case[k]) for k in ("store", "init", "dst")]
            item = {"in": codec.store(x, eb[0]).clone(), "n_bytes": 4 * x.numel(), "eb1": eb[1], "src": clients[i]}
            first.append(dict(item, out=outs[2 * i], out_size=sizes[2 * i:]))
            second.append(dict(item, out=outs[2 * i + 1], out_size=sizes[2 * i + 1:], eb2=eb[2]))
        return dict(state, clients=clients, first=first, second=second)

    x = xs[0]
    n = 4 * x.numel()
    codec.reserve(-(-n // 16384))
    state.update(n=n, sizes=torch.zeros(8, dtype=torch.int64, device="cuda"),
                 minmax=codec.INOA_find_range_device(x))
    eb = {k: _scaled(case, x, case[k]) for k in ("store", "init", "dst") if k in case}
    rel = {k: float(storage.f32(case[k])) for k in eb}
    state.update(eb=eb, rel=rel)

    def stream():
        return torch.zeros(max_stream_bytes(n), dtype=torch.uint8, device="cuda")

    if op in ("store", "flow", "step"):
        state.update(x=x, stored=stream())
        if op != "store":
            state.update(init=stream(), resi=stream(), client=torch.zeros_like(x), final=torch.zeros_like(x))
        return state
    stored = codec.store(x, eb["store"]).clone()
    if op == "load":
        state.update(stored=stored, out=torch.zeros_like(x))
    elif op == "init_send":
        state.update(stored=stored, init=stream())
    elif op == "resi_send":
        state.update(stored=stored, resi=stream())
    else:
        init = codec.init_send(stored, eb["init"]).clone()
        if op == "init_recv":
            state.update(init=init, out=torch.zeros_like(x))
        else:
            state.update(client=codec.init_recv(init), resi=codec.resi_send(stored, eb["init"], eb["dst"]).clone(),
                         out=torch.zeros_like(x))
    return state


# ------------------------------------------------------------------ one pass
def run(s):
    c, case = s["codec"], s["case"]
    op, mode = case["op"], case["mode"]
    if op == "chain":
        chain = s["chain"]
        chain.replay()
        return {"recon": chain.recon, "streams": chain.streams, "sizes": chain.sizes, "first_bad": chain.first_bad}
    if op == "batch_store":
        c.batch("store", s["items"])
        return {"streams": s["arena"], "sizes": s["sizes"]}
    if op == "batch_serve":
        c.batch("init_send_apply", s["first"])
        c.batch("resi_send_apply", s["second"])
        return {"streams": s["arena"], "sizes": s["sizes"], "clients": s["clients"]}
    n, sz, mm, eb, rel = s["n"], s["sizes"], s["minmax"], s["eb"], s["rel"]
    if op == "store":
        if mode == "noa":
            c.INOA_find_range_device(s["x"], mm)
            c.server_encode_noa(s["x"], n, s["stored"], sz, mm, rel["store"])
            return {"stored": s["stored"], "size": sz, "range": mm}
        bound = eb["store"]
        if mode == "host":
            lo, hi = c.INOA_find_range(s["x"])
            bound = float(storage.noa_scale(case["store"], storage.value_range(lo, hi)))
        c.server_encode(s["x"], n, s["stored"], sz, bound)
        return {"stored": s["stored"], "size": sz}
    if op == "load":
        c.server_decode(s["stored"], s["out"], sz)
        return {"out": s["out"], "size": sz}
    if op == "init_send":
        if mode == "noa":
            c.s2c_encode_noa(s["stored"], s["init"], sz, mm, rel["init"], n)
        else:
            c.s2c_encode(s["stored"], s["init"], sz, eb["init"], n)
        return {"init": s["init"], "size": sz}
    if op == "init_recv":
        c.client_decode(s["init"], s["out"], sz)
        return {"out": s["out"], "size": sz}
    if op == "resi_send":
        if mode == "noa":
            c.residual_encode_noa(s["stored"], s["resi"], sz, mm, rel["init"], rel["dst"], n)
        else:
            c.residual_encode(s["stored"], s["resi"], sz, eb["init"], eb["dst"], n)
        return {"resi": s["resi"], "size": sz}
    if op == "resi_recv":
        c.residual_apply(s["client"], n, s["resi"], s["out"], sz)
        return {"out": s["out"], "size": sz}
    # flow: the exchange call by call; step: the sends fused with the client's side
    c.INOA_find_range_device(s["x"], mm)
    c.server_encode_noa(s["x"], n, s["stored"], sz[0:], mm, rel["store"])
    if op == "flow":
        c.s2c_encode_noa(s["stored"], s["init"], sz[1:], mm, rel["init"], n)
        c.client_decode(s["init"], s["client"], sz[2:])
        c.residual_encode_noa(s["stored"], s["resi"], sz[3:], mm, rel["init"], rel["dst"], n)
        c.residual_apply(s["client"], n, s["resi"], s["final"], sz[4:])
        return {k: s[k] for k in ("stored", "init", "resi", "client", "final", "sizes", "minmax")}
    c.s2c_encode_apply_noa(s["stored"], s["init"], sz[1:], mm, rel["init"], n, s["client"])
    c.residual_encode_apply_noa(s["stored"], s["resi"], sz[2:], mm, rel["init"], rel["dst"], n, s["client"])
    return {k: s[k] for k in ("stored", "init", "resi", "client", "sizes", "minmax")}


# ------------------------------------------------------------------ what a pass cannot do without
def _stream_bytes(words, kind, bound, mode):
    """About what a stream takes: the bits that the differences of neighbours need at the bound, and half a bit for
    the bitmaps."""
    span, step = {"sinusoid": (6.0, 0.05), "outliers": (2e6, 0.05), "grf": (8.0, 0.05), "white": (2.0, 0.7)}[kind]
    width = bound if mode == "abs" else bound * span
    return words * min(32.0, math.log2(1 + 2 * step / width) + 0.2) / 8


def work(case):
    op = case["op"]
    if op == "chain":
        w = case["rows"] * case["cols"]
        total = 0.0
        for i, b in enumerate(CHAIN_STEPS):
            kept = max(k for k in CHAIN_STORE if k <= b)
            sent = _stream_bytes(w, "grf", b, "noa")
            # stored stream in, request stream out and in, the client's floats in (not at first) and out, the check
            total += _stream_bytes(w, "grf", kept, "noa") + 2 * sent + 4 * w * (4 if i else 3)
        return {"bytes": total, "flops": 0}
    if "fields" in case:
        total = 0.0
        for i, w in enumerate(_batch_sizes(case)):
            kind = KINDS[i % 3]
            if op == "batch_store":
                total += 4 * w + sum(_stream_bytes(w, kind, b, "noa") for b in BATCH_STORE)
            else:
                total += 2 * _stream_bytes(w, kind, case["store"], "noa") + 12 * w
                total += sum(_stream_bytes(w, kind, case[k], "noa") for k in ("init", "dst"))
        return {"bytes": total, "flops": 0}
    w = case["words"]
    stored, init, resi = (_stream_bytes(w, case["kind"], case[k], case["mode"]) if k in case else 0.0
                          for k in ("store", "init", "dst"))
    ranged = 4 * w if case["mode"] != "abs" else 0
    total = {"store": ranged + 4 * w + stored, "load": stored + 4 * w, "init_send": stored + init,
             "init_recv": init + 4 * w, "resi_send": stored + resi, "resi_recv": resi + 8 * w,
             "flow": 8 * w + 3 * stored + 2 * init + 4 * w + 2 * resi + 8 * w,
             "step": 8 * w + 3 * stored + init + 4 * w + resi + 8 * w}[op]
    return {"bytes": total, "flops": 0}


# ------------------------------------------------------------------ the decoded values, in 64 bits
def _grid(bound):
    """Width of a bound's bins and the magnitude from which values are kept as they are."""
    e = math.frexp(bound)[1]  # 2^(e-1) <= bound < 2^e
    return math.ldexp(1.0, e), math.ldexp(1.0, e + 23)


def _rounded(x, bound):
    """A request's values: the nearest multiple of the bin width, halves away from zero."""
    width, whole = _grid(bound)
    y = torch.floor(x.abs() / width + 0.5) * width * torch.sign(x)
    return torch.where(x.abs() < whole, y, x)


def exact(case, seed):
    op = case["op"]
    if op in ("batch_store", "init_send", "resi_send") or (op == "store" and case["mode"] != "noa"):
        return None  # streams and sizes: bytes and whole numbers
    xs = _inputs(case, seed)
    if op == "store":
        return {"stored": None, "size": None, "range": torch.stack((xs[0].min(), xs[0].max())).double()}
    if op == "chain":
        x = xs[0].double()
        return {"recon": [_rounded(x, _scaled(case, xs[0], b)) for b in CHAIN_STEPS], "streams": None, "sizes": None,
                "first_bad": None}
    if op == "batch_serve":
        return {"streams": None, "sizes": None,
                "clients": [_rounded(x.double(), _scaled(case, x, case["dst"])) for x in xs]}
    x = xs[0]
    if op == "load":
        width, whole = _grid(_scaled(case, x, case["store"]) / 2)
        d = x.double()
        return {"out": torch.where(d.abs() < whole, torch.trunc(d / width) * width, d), "size": None}
    first = _rounded(x.double(), _scaled(case, x, case["init"]))
    if op == "init_recv":
        return {"out": first, "size": None}
    second = _rounded(x.double(), _scaled(case, x, case["dst"]))
    if op == "resi_recv":
        return {"out": second, "size": None}
    got = dict(stored=None, init=None, resi=None, sizes=None, minmax=torch.stack((x.min(), x.max())).double())
    return dict(got, client=first, final=second) if op == "flow" else dict(got, client=second)
