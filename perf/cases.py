"""Measured cases of the PFP BWT library: what its users call, over the sizes
that they call it with.

A case is a dict of plain values.  ``call`` names the entry point:

  device   Storage.pfp_bwt_device: one text, text and BWT in device memory
  host     Storage.pfp_bwt_into: one text, pinned host buffers
  bytes    Storage.libcubwt_bwt: one host text with any byte values
  batch    Storage.pfp_bwt_batch_device: many texts in one call
  serve    Server.submit / wait: jobs of mixed sizes submitted in one burst
  inverse  Storage.unbwt_device: BWT and primary index back to the text

and ``text`` the kind of content, as in the package's workloads module:

  dna      mutated copies of a uniform ACGT base (0.1 % substitutions,
           0.01 % indels), coded 2..5
  versions successive versions of an order-3 Markov text over bytes 32..127,
           blocks of 1..64 bytes replaced at ``rate`` per byte

Texts are made on the GPU from the seed alone and cut to exactly ``bytes``.
One storage object (and one server) is kept for the process and reused, as
the library asks its users to do.
"""
from __future__ import annotations

import importlib
import math

import numpy as np
import torch

PKG = "masterarbeit_parallele_konstruktion_der_burrows-wheeler-transformation_auf_der_gpu_gb300"
KiB, MiB = 1 << 10, 1 << 20


# ---- cases --------------------------------------------------------------------

def listed() -> list[dict]:
    return [
        # one small text per call: the median job of the serving mix is 64 KiB, the smallest 4 KiB;
        # launches and host round trips are what it pays for
        dict(name="dna 24 KiB", call="device", text="dna", bytes=24 * KiB + 3, copies=16, W=5, P=16, small=False),
        # the small benchmark text: 32 copies of 256 KiB
        dict(name="dna 8 MiB", call="device", text="dna", bytes=8 * MiB, copies=32, W=5, P=16, small=False),
        # the headline text: 128 copies of 4 MiB
        dict(name="dna 512 MiB", call="device", text="dna", bytes=512 * MiB, copies=128, W=5, P=16, small=False),
        # the same kind of text with the long-window small-alphabet parameters
        dict(name="dna 512 MiB W35", call="device", text="dna", bytes=512 * MiB, copies=128, W=35, P=81, small=True),
        # large-alphabet versioned text: 128 versions of 2 MiB
        dict(name="versions 256 MiB", call="device", text="versions", bytes=256 * MiB, copies=128, rate=1e-4, W=5,
             P=23, small=False),
        # a log- or source-like file of the size of the thesis' 102 MB files: little repetition, a large dictionary
        dict(name="versions 102 MB", call="device", text="versions", bytes=102_000_001, copies=3, rate=2e-3, W=5,
             P=13, small=False),
        # 4096 texts of uneven lengths in one call
        dict(name="batch 4096", call="batch", text="dna", bytes=512 * MiB, texts=4096, W=5, P=16, small=False),
        # a small batch, as the serving loop forms from the jobs that are waiting
        dict(name="batch 24", call="batch", text="dna", bytes=3 * MiB + 17, texts=24, W=5, P=16, small=False),
        # host to host through pinned buffers, as a program that reads files calls it
        dict(name="host 96 MiB", call="host", text="dna", bytes=96 * MiB + 5, copies=48, W=5, P=14, small=True),
        # a caller of libcubwt: pageable host buffers, any byte values
        dict(name="bytes 16 MiB", call="bytes", text="versions", bytes=16 * MiB + 1, copies=16, rate=1e-3, W=5, P=16,
             small=False),
        # a burst of serving jobs: 99 small ones and one large
        dict(name="serve 100", call="serve", text="dna", bytes=80 * MiB, texts=100, W=5, P=16, small=False),
        # decoding: the text back from its BWT
        dict(name="inverse 128 MiB", call="inverse", text="dna", bytes=128 * MiB + 11, copies=64, W=5, P=16,
             small=False),
    ]


def draw(rng) -> dict:
    """One more case: the listed calls, sizes spread over the logarithm of their range."""
    def size(lo, hi):
        n = int(math.exp(rng.uniform(math.log(lo), math.log(hi))))
        return max(lo, min(hi, n | rng.randrange(2)))

    call = rng.choice(["device", "device", "device", "device", "batch", "host", "bytes", "serve", "inverse"])
    case = dict(call=call, text="dna", W=5, P=16, small=False)
    if call in ("device", "host", "bytes", "inverse"):
        hi = {"device": 512 * MiB, "host": 256 * MiB, "bytes": 64 * MiB, "inverse": 256 * MiB}[call]
        case["bytes"] = size(4 * KiB, hi)
        case["copies"] = max(1, min(rng.choice([2, 8, 16, 32, 64, 128]), case["bytes"] // 1024))
        if call == "bytes" or rng.random() < 0.4:
            # large alphabets: sizes and repetition of the versioned text (fewer versions: smaller texts)
            case["text"] = "versions"
            case["bytes"] = min(case["bytes"], 256 * MiB)
            case["copies"] = min(case["copies"], 128)
            if case["copies"] < 16:
                case["bytes"] = min(case["bytes"], 102_000_001)
            case["rate"] = rng.choice([1e-4, 1e-3, 2e-3])
        if call in ("device", "host"):
            if case["text"] == "dna":
                case["W"], case["P"], case["small"] = rng.choice(
                    [(5, 16, False), (5, 16, True), (5, 14, True), (5, 23, True), (35, 81, True)])
                if case["copies"] < 16:
                    case["bytes"] = min(case["bytes"], 128 * MiB)
            else:
                case["P"] = rng.choice([11, 13, 14, 16, 23])
    elif call == "batch":
        case["bytes"] = size(256 * KiB, 512 * MiB)
        case["texts"] = max(2, min(4096, int(case["bytes"] / rng.uniform(32 * KiB, 160 * KiB))))
    else:
        case["bytes"] = size(4 * MiB, 80 * MiB)
        case["texts"] = rng.randrange(8, 101)
    return case


def work(case: dict) -> dict:
    """Every text byte read once and every BWT byte written once."""
    return {"bytes": 2.0 * case["bytes"], "flops": 0.0}


# ---- texts --------------------------------------------------------------------

class _Gen:
    """Random numbers on the GPU and on the host, both from the seed."""

    def __init__(self, seed: int):
        self.t = torch.Generator(device="cuda")
        self.t.manual_seed(seed)
        self.n = np.random.default_rng(seed)

    def ints(self, lo, hi, n, dtype=torch.int64):
        return torch.randint(lo, hi, (n,), generator=self.t, device="cuda", dtype=dtype)

    def rand(self, n):
        return torch.rand(n, generator=self.t, device="cuda")


def _substitute(g: _Gen, seq: torch.Tensor, rate: float) -> torch.Tensor:
    hit = (g.rand(seq.numel()) < rate).to(torch.uint8)
    shift = g.ints(1, 4, seq.numel(), torch.uint8) * hit                # a new base differs from the old one
    return (seq - 2 + shift) % 4 + 2


def _indels(g: _Gen, seq: torch.Tensor, rate: float) -> torch.Tensor:
    n = seq.numel()
    k = int(g.n.binomial(n, rate))
    if k == 0:
        return seq
    pos, ln, ins = g.ints(0, n, k), g.ints(1, 11, k), g.ints(0, 2, k)
    step = torch.zeros(n + 16, dtype=torch.int32, device="cuda")         # running number of open deletions
    one = (1 - ins).to(torch.int32)
    step.index_add_(0, pos, one)
    step.index_add_(0, pos + ln, -one)
    times = (torch.cumsum(step, 0)[:n] <= 0).to(torch.int64)             # how often each byte is written
    extra = torch.zeros(n, dtype=torch.int64, device="cuda")
    extra.index_add_(0, pos, ln * ins)
    out = torch.repeat_interleave(seq, times + extra)
    # the inserted bytes follow the byte they were repeated from: replace them by uniform bases
    first = torch.cumsum(times + extra, 0) - extra
    at = torch.repeat_interleave(first, extra)
    base = torch.cumsum(extra, 0) - extra
    at = at + torch.arange(at.numel(), device="cuda") - torch.repeat_interleave(base, extra)
    out[at] = g.ints(2, 6, at.numel(), torch.uint8)
    return out


def _dna(g: _Gen, n: int, copies: int) -> torch.Tensor:
    base = g.ints(2, 6, -(-n // copies), torch.uint8)
    parts, have = [], 0
    while have < n:
        p = _indels(g, _substitute(g, base, 1e-3), 1e-4)
        parts.append(p)
        have += p.numel()
    return torch.cat(parts)[:n].contiguous()


def _markov(g: _Gen, n: int) -> torch.Tensor:
    """n symbols 0..95 of order-3 Markov chains whose rows are Dirichlet(0.1)
    (contexts share 8192 rows), run side by side and laid end to end."""
    rows = 8192
    chains = max(64, min(16384, n // 1024))
    steps = -(-n // chains)
    cdf = torch.from_numpy(np.cumsum(g.n.dirichlet(np.full(96, 0.1), rows), 1).astype(np.float32)).cuda()
    a, b, c = (g.ints(0, 96, chains) for _ in range(3))
    out = torch.empty((steps, chains), dtype=torch.uint8, device="cuda")
    for i in range(steps):
        row = cdf[(a * 7919 + b * 104_729 + c * 31) % rows]
        s = torch.searchsorted(row, g.rand(chains).unsqueeze(1)).squeeze(1).clamp_(max=95)
        out[i] = s
        a, b, c = b, c, s
    return out.t().reshape(-1)[:n].contiguous()


def _versions(g: _Gen, n: int, copies: int, rate: float) -> torch.Tensor:
    base = -(-n // copies)
    fresh = max(4096, base // 2)
    both = _markov(g, base + fresh) + 32
    cur, pool = both[:base].clone(), both[base:]
    out = [cur]
    for _ in range(copies - 1):
        cur = cur.clone()
        k = int(g.n.binomial(base, rate))
        if k:
            ln = g.ints(1, 65, k)
            at, src = g.ints(0, base, k), g.ints(0, fresh - 64, k)
            off = torch.arange(int(ln.sum()), device="cuda") - torch.repeat_interleave(torch.cumsum(ln, 0) - ln, ln)
            at, src = torch.repeat_interleave(at, ln) + off, torch.repeat_interleave(src, ln) + off
            # blocks may meet: the byte with the largest source position stays
            want = torch.full((base + 64,), -1, dtype=torch.int64, device="cuda")
            want.scatter_reduce_(0, at, src, "amax")
            want = want[:base]
            cur = torch.where(want >= 0, pool[want.clamp(min=0)], cur)
        out.append(cur)
    return torch.cat(out)[:n].contiguous()


def _text(case: dict, g: _Gen) -> torch.Tensor:
    if case["text"] == "dna":
        return _dna(g, case["bytes"], case["copies"])
    t = _versions(g, case["bytes"], case["copies"], case["rate"])
    if case["call"] == "bytes":
        values = np.sort(np.concatenate([[0, 255], 1 + g.n.permutation(254)[:94]])).astype(np.uint8)
        t = torch.from_numpy(values).cuda()[t.long() - 32]
    return t


def _lengths(case: dict, g: _Gen) -> np.ndarray:
    """Log-normal text lengths (sigma 1.2) that sum to the case's bytes; a
    burst of serving jobs holds one large text of four fifths of them."""
    k, total = case["texts"], case["bytes"]
    big = total * 4 // 5 if case["call"] == "serve" else 0
    rest, m = total - big, k - (1 if big else 0)
    w = g.n.lognormal(0.0, 1.2, m)
    lens = np.maximum(1, (w * (rest / w.sum())).astype(np.int64))
    lens[int(np.argmax(lens))] += rest - int(lens.sum())
    if big:
        lens = np.insert(lens, m // 2, big)
    return lens


def _texts(case: dict, g: _Gen) -> tuple[torch.Tensor, np.ndarray]:
    """Texts of uneven lengths, each 8..64 mutated copies of its own base."""
    lens = _lengths(case, g)
    parts = []
    for n in lens.tolist():
        base = g.ints(2, 6, max(1, n // int(g.n.integers(8, 65))), torch.uint8)
        parts.append(base.repeat(-(-n // base.numel()))[:n])
    t = torch.cat(parts)
    offsets = np.zeros(len(lens) + 1, dtype=np.int64)
    np.cumsum(lens, out=offsets[1:])
    return _substitute(g, t, 1e-3), offsets


# ---- preparing and running ----------------------------------------------------

_KEPT: dict = {}


def _storage():
    if "storage" not in _KEPT:
        _KEPT["storage"] = importlib.import_module(PKG).Storage()
    return _KEPT["storage"]


def _server():
    if "server" not in _KEPT:
        _KEPT["server"] = importlib.import_module(PKG).Server()
    return _KEPT["server"]


def prepare(case: dict, seed: int) -> dict:
    g = _Gen(seed)
    call = case["call"]
    s = {"case": dict(case)}
    if call in ("batch", "serve"):
        t, s["offsets"] = _texts(case, g)
    else:
        t = _text(case, g)
    if call == "serve":
        s["text"], s["out"] = t.cpu().numpy(), np.empty(case["bytes"], np.uint8)
        s["server"] = _server()
    elif call == "host":
        s["text"] = t.cpu().pin_memory().numpy()
        s["out"] = torch.empty(case["bytes"], dtype=torch.uint8).pin_memory().numpy()
    elif call == "bytes":
        s["text"] = t.cpu().numpy()
    else:
        s["text"], s["out"] = t, torch.empty_like(t)
    if call != "serve":
        s["storage"] = _storage()
    if call == "inverse":
        torch.cuda.synchronize()
        L = torch.empty_like(t)
        s["storage"].pfp_bwt_device(t.data_ptr(), L.data_ptr(), case["bytes"], case["W"], case["P"], case["small"])
        s["bwt"], s["primary"] = L, s["storage"].stats()["primary_index"]
        del s["text"]
    torch.cuda.synchronize()             # the storage has a stream of its own
    return s


def run(s: dict):
    case, call = s["case"], s["case"]["call"]
    W, P, small = case["W"], case["P"], case["small"]
    if call == "device":
        s["storage"].pfp_bwt_device(s["text"].data_ptr(), s["out"].data_ptr(), case["bytes"], W, P, small)
    elif call == "host":
        s["storage"].pfp_bwt_into(s["text"], s["out"], W, P, small)
    elif call == "bytes":
        L, index = s["storage"].libcubwt_bwt(s["text"])
        return {"bwt": L, "index": index}
    elif call == "batch":
        s["storage"].pfp_bwt_batch_device(s["text"].data_ptr(), s["offsets"], s["out"].data_ptr(), W, P, small)
    elif call == "serve":
        o, text, out, server = s["offsets"].tolist(), s["text"], s["out"], s["server"]
        tickets = [server.submit(text[a:b], W, P, small, out=out[a:b]) for a, b in zip(o, o[1:])]
        for ticket in tickets:
            server.result(ticket)
            server.release(ticket)
    else:
        s["storage"].unbwt_device(s["bwt"].data_ptr(), s["out"].data_ptr(), case["bytes"], s["primary"])
    return {"out": s["out"]}


# ---- expected values ------------------------------------------------------------

def _suffix_order(t: torch.Tensor) -> torch.Tensor:
    """Suffix array by prefix doubling with torch sorts; a suffix sorts before
    the longer ones that it starts."""
    n = t.numel()
    rank, h = t.long() + 1, 1
    while True:
        nxt = torch.zeros_like(rank)
        if h < n:
            nxt[:n - h] = rank[h:]
        key, order = torch.sort(rank * (max(n, 256) + 2) + nxt)
        fresh = torch.ones_like(key)
        fresh[1:] = (key[1:] != key[:-1]).long()
        rank = torch.empty_like(rank)
        rank[order] = torch.cumsum(fresh, 0)
        if int(rank.max()) == n or h >= n:
            return order
        h *= 2


def _bwt(t: torch.Tensor) -> torch.Tensor:
    return t[(_suffix_order(t) - 1) % t.numel()]


def exact(case: dict, seed: int):
    """The BWT from the definition (the text itself for the inverse), with
    plain torch; None where that takes long."""
    call = case["call"]
    if call != "inverse" and (case["bytes"] > 128 * MiB or case.get("texts", 0) > 128):
        return None
    g = _Gen(seed)
    if call in ("batch", "serve"):
        t, o = _texts(case, g)
        return {"out": torch.cat([_bwt(t[a:b]) for a, b in zip(o[:-1].tolist(), o[1:].tolist())])}
    t = _text(case, g)
    if call == "inverse":
        return {"out": t}
    order = _suffix_order(t)
    L = t[(order - 1) % t.numel()]
    if call != "bytes":
        return {"out": L}
    # libcubwt: the last byte first, the row of the whole text left out; its number is the index
    row = int((order == 0).nonzero())
    return {"bwt": torch.cat([t[-1:], L[:row], L[row + 1:]]), "index": row + 1}
