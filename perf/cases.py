"""The calls this library is timed on: constructions (one text, a batch, host to host, served), and
the operations on their results (LCP array, inverse BWT, suffix array check).

Every text is made on the GPU from the seed, with the shapes of ``sadcs_b200.workloads``: uniform
bytes (8-bit codes), natural-language-like text (6 bits), protein-like text (5 bits), {A,C,G,T} text
with and without mutated repeats (2 bits), and successive versions of one document, whose long
common prefixes the sample ranking has to double through.
"""
import math

import numpy as np
import torch

import sadcs_b200

MIB = 1 << 20


def listed():
    return [
        # One short document per call (an editor, a query's text): launches and latency count.
        {"name": "text_64k", "op": "build", "text": "natural", "n": 65_521},
        # Incompressible bytes of the reference's CPU-runnable size: no repeats, the widest codes.
        {"name": "uniform_8m", "op": "build", "text": "uniform", "n": 8 * MIB},
        # A text collection: the benchmark's 256 MiB natural-language-like text.
        {"name": "natural_256m", "op": "build", "text": "natural", "n": 256 * MIB},
        # A genome with repeats, the largest text an int32 suffix array takes.
        {"name": "genome_2g", "op": "build", "text": "genome", "n": 2**31 - 1025},
        # A compressor's use: the BWT alone (no suffix array), of a protein database, ragged size.
        {"name": "protein_bwt_100m", "op": "bwt", "text": "protein", "n": 100_000_007},
        # Versions of one document (backups, page histories): long repeats.
        {"name": "versions_48m", "op": "build", "text": "versions", "n": 48 * MIB + 11},
        # Many texts in one construction: the benchmark's batch (DNA, protein, uniform in turn).
        {"name": "batch_4096", "op": "batch", "count": 4096, "lo": 1 << 10, "hi": 4 * MIB},
        # The call of a program that holds its text in host memory, page-locked buffers.
        {"name": "host_64m", "op": "host", "text": "natural", "n": 64 * MIB + 5},
        # A burst of requests to the server: small ones are built together.
        {"name": "serve_burst", "op": "serve", "count": 48, "lo": 4 << 10, "hi": 16 * MIB},
        # An index's next step after the suffix array: its LCP array.
        {"name": "lcp_128m", "op": "lcp", "text": "natural", "n": 128 * MIB},
        # Decompression: the text back from its BWT.
        {"name": "unbwt_64m", "op": "unbwt", "text": "natural", "n": 64 * MIB + 3},
        # A suffix array that was read from a file or made elsewhere: verified, then its BWT taken.
        {"name": "check_128m", "op": "check", "text": "genome", "n": 128 * MIB + 1},
    ]


# The largest text of a drawn case, by operation (a drawn case costs no more than genome_2g).
_DRAW_MAX = {"build": 512 * MIB, "bwt": 256 * MIB, "host": 128 * MIB, "lcp": 256 * MIB, "unbwt": 64 * MIB,
             "check": 256 * MIB}
_DRAW_MIN = {"build": 2 << 10, "bwt": 16 << 10, "host": 64 << 10, "lcp": 64 << 10, "unbwt": 64 << 10,
             "check": 64 << 10}


def _log_uniform(rng, lo, hi):
    return int(math.exp(rng.uniform(math.log(lo), math.log(hi))))


def draw(rng):
    # the constructions carry most calls
    op = rng.choice(["build", "build", "build", "build", "bwt", "batch", "host", "serve", "lcp", "unbwt", "check"])
    if op == "batch":
        lo = _log_uniform(rng, 256, 16 << 10)
        return {"op": "batch", "count": _log_uniform(rng, 3, 2048), "lo": lo, "hi": _log_uniform(rng, 32 << 10, MIB)}
    if op == "serve":
        return {"op": "serve", "count": rng.randint(4, 60), "lo": _log_uniform(rng, 1 << 10, 64 << 10),
                "hi": _log_uniform(rng, 128 << 10, 16 * MIB)}
    text = rng.choice(["natural", "uniform", "genome", "protein", "versions"])
    top = min(_DRAW_MAX[op], 64 * MIB) if text == "versions" else _DRAW_MAX[op]
    return {"op": op, "text": text, "n": _log_uniform(rng, _DRAW_MIN[op], top) | rng.randint(0, 1)}


# ---- texts ---------------------------------------------------------------------------------------

_CHUNK = 32 * MIB  # characters made at a time, so that temporaries stay small beside the text
_DNA = b"ACGT"
_AMINO = b"ACDEFGHIKLMNPQRSTVWY"
_AMINO_FREQ = (8.25, 1.37, 5.45, 6.75, 3.86, 7.07, 2.27, 5.96, 5.84, 9.66, 2.42, 4.06, 4.70, 3.93, 5.53, 6.56, 5.34,
               6.87, 1.08, 2.92)


def _bytes(s):
    return torch.tensor(list(s), dtype=torch.uint8, device="cuda")


def _letters(g, out, letters, weights):
    """out filled with independent letters of the given frequencies."""
    cdf = torch.tensor(weights, dtype=torch.float64).cumsum(0)
    cdf = (cdf / cdf[-1])[:-1].to(torch.float32).cuda()
    table = _bytes(letters)
    for s in range(0, out.numel(), _CHUNK):
        u = torch.rand(min(_CHUNK, out.numel() - s), device="cuda", generator=g)
        out[s:s + u.numel()] = table[torch.bucketize(u, cdf, right=True, out_int32=True)]


def _uniform(g, out):
    for s in range(0, out.numel(), 4 * _CHUNK):
        e = min(s + 4 * _CHUNK, out.numel())
        out[s:e] = torch.randint(0, 256, (e - s,), device="cuda", generator=g, dtype=torch.uint8)


def _dna(g, out):
    _letters(g, out, _DNA, (0.295, 0.205, 0.205, 0.295))


def _protein(g, out):
    _letters(g, out, _AMINO, _AMINO_FREQ)


def _genome(g, out):
    """Two thirds independent letters, then mutated copies of 1 MiB pieces of them: 1% substitutions
    and 0.1% insertions and deletions."""
    n = out.numel()
    base = (2 * n) // 3
    _dna(g, out[:base])
    if base < 2:
        _dna(g, out[base:])
        return
    letters = _bytes(_DNA)
    piece = min(MIB, max(1, base // 2))
    for s in range(base, n, 16 * piece):
        m = min(16 * piece, n - s)
        pieces = -(-m // piece)
        starts = torch.randint(0, max(1, base - piece - piece // 50), (pieces, 1), device="cuda", generator=g)
        event = torch.rand((pieces, piece), device="cuda", generator=g)
        gap = torch.randint(1, 11, (pieces, piece), device="cuda", generator=g)
        step = torch.where(event < 0.0005, gap + 1, torch.ones_like(gap))  # deletions skip 1-10 characters
        insert = (event >= 0.0005) & (event < 0.001)
        step = torch.where(insert, torch.zeros_like(step), step)
        at = (starts + step.cumsum(1)).clamp_(max=base - 1)
        copy = out[at.reshape(-1)[:m]]
        fresh = (torch.rand(m, device="cuda", generator=g) < 0.01) | insert.reshape(-1)[:m]
        other = letters[torch.randint(0, 4, (m,), device="cuda", generator=g)]
        out[s:s + m] = torch.where(fresh, other, copy)


def _natural(g, out):
    """Words of 2-12 lowercase letters drawn by Zipf's law from 50,000, spaces between, a full stop
    and a line end after 5% of them, 2% capitalised."""
    vocabulary = 50_000
    lengths = torch.randint(2, 13, (vocabulary,), device="cuda", generator=g)
    first = lengths.cumsum(0) - lengths
    letters = torch.randint(ord("a"), ord("z") + 1, (int(lengths.sum()),), device="cuda", generator=g,
                            dtype=torch.uint8)
    cdf = (1.0 / torch.arange(1, vocabulary + 1, dtype=torch.float64, device="cuda") ** 1.1).cumsum(0)
    cdf = (cdf / cdf[-1])[:-1].to(torch.float32)
    filled, n = 0, out.numel()
    while filled < n:
        want = min(_CHUNK, n - filled)
        count = want // 6 + 64
        word = torch.bucketize(torch.rand(count, device="cuda", generator=g), cdf, right=True)
        stop = torch.rand(count, device="cuda", generator=g) < 0.05
        capital = torch.rand(count, device="cuda", generator=g) < 0.02
        size = lengths[word] + 1 + stop
        ends = size.cumsum(0)
        owner = torch.repeat_interleave(torch.arange(count, device="cuda"), size)
        inside = torch.arange(owner.numel(), device="cuda") - (ends - size)[owner]
        letter = inside < lengths[word][owner]
        chunk = letters[torch.where(letter, first[word][owner] + inside, torch.zeros_like(inside))]
        chunk = torch.where(capital[owner] & (inside == 0), chunk - 32, chunk)
        after = inside - lengths[word][owner]
        dot = stop[owner]
        chunk = torch.where(~letter & ~dot, torch.full_like(chunk, 32), chunk)
        chunk = torch.where(~letter & dot & (after == 0), torch.full_like(chunk, 46), chunk)
        chunk = torch.where(~letter & dot & (after == 1), torch.full_like(chunk, 10), chunk)
        take = min(want, chunk.numel())
        out[filled:filled + take] = chunk[:take]
        filled += take


def _versions(g, out):
    """A document of natural text (up to 1 MiB), then versions of it: each changes 32 places of the one
    before."""
    size = min(MIB, max(64, out.numel() // 16))
    page = torch.empty(size, dtype=torch.uint8, device="cuda")
    _natural(g, page)
    for s in range(0, out.numel(), size):
        out[s:s + size] = page[:out.numel() - s]
        at = torch.randint(0, size, (32,), device="cuda", generator=g)
        page[at] = torch.randint(ord("a"), ord("z") + 1, (32,), device="cuda", generator=g, dtype=torch.uint8)


_TEXTS = {"natural": _natural, "uniform": _uniform, "dna": _dna, "genome": _genome, "protein": _protein,
          "versions": _versions}


def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _text(kind, n, seed):
    out = torch.empty(n, dtype=torch.uint8, device="cuda")
    _TEXTS[kind](_generator(seed), out)
    torch.cuda.empty_cache()  # the temporaries' memory, for the context
    return out


def _lengths(case):
    """Log-uniform lengths in [lo, hi]; the case's sizes do not depend on the seed."""
    r = np.random.default_rng([case["count"], case["lo"], case["hi"]])
    return np.exp(r.uniform(np.log(case["lo"]), np.log(case["hi"]), case["count"])).astype(np.int64)


def _many(case, seed):
    """The texts of a batch or a burst back to back: DNA, protein-like and uniform bytes in turn."""
    lengths = _lengths(case)
    g = _generator(seed)
    out = torch.empty(int(lengths.sum()), dtype=torch.uint8, device="cuda")
    at = 0
    for j, n in enumerate(lengths.tolist()):
        (_dna, _protein, _uniform)[j % 3](g, out[at:at + n])
        at += n
    torch.cuda.empty_cache()
    return lengths, out


# ---- the calls -----------------------------------------------------------------------------------

def _u32(n):
    return torch.empty(n, dtype=torch.int32, device="cuda")


def _u8(n):
    return torch.empty(n, dtype=torch.uint8, device="cuda")


def _pinned(n, dtype):
    """Page-locked host memory of n entries, as the array the host calls take."""
    raw = torch.empty(n * np.dtype(dtype).itemsize, dtype=torch.uint8, pin_memory=True)
    return raw.numpy().view(dtype)


def prepare(case, seed):
    op = case["op"]
    if op == "serve":
        lengths, device = _many(case, seed)
        total = int(lengths.sum())
        text = _pinned(total, np.uint8)
        torch.from_numpy(text).copy_(device)
        server = sadcs_b200.Server(memory_budget=16 << 30, workers=3, small_limit=64 * MIB, batch_bytes=512 * MIB,
                                   batch_texts=4096)
        at = np.concatenate([[0], np.cumsum(lengths)]).tolist()
        return {"op": op, "server": server, "at": at, "text": text, "sa": _pinned(total, np.uint32),
                "bwt": _pinned(total, np.uint8)}
    if op == "batch":
        lengths, text = _many(case, seed)
        total = int(lengths.sum())
        state = {"op": op, "lengths": lengths, "text": text, "sa": _u32(total), "bwt": _u8(total),
                 "context": sadcs_b200.Context(total, max_texts=len(lengths))}
        torch.cuda.synchronize()
        return state
    n = case["n"]
    text = _text(case["text"], n, seed)
    state = {"op": op, "n": n, "text": text}
    if op == "host":
        state["text"] = _pinned(n, np.uint8)
        torch.from_numpy(state["text"]).copy_(text)
        state.update(sa=_pinned(n, np.uint32), bwt=_pinned(n, np.uint8), context=sadcs_b200.Context(n))
    elif op in ("build", "bwt"):
        state.update(sa=_u32(n) if op == "build" else None, bwt=_u8(n), context=sadcs_b200.Context(n))
    else:  # operations on a construction's results
        sa, bwt = _u32(n), _u8(n)
        torch.cuda.synchronize()
        with sadcs_b200.Context(n) as context:
            primary = sadcs_b200.build_device(text.data_ptr(), n, sa.data_ptr(), bwt.data_ptr(), context)
        if op == "lcp":
            state.update(sa=sa, lcp=_u32(n))
        elif op == "unbwt":
            state.update(bwt=bwt, primary=primary, out=_u8(n))
        else:
            state.update(sa=sa, bwt=bwt)
    torch.cuda.synchronize()
    return state


def run(state):
    op = state["op"]
    if op == "build":
        primary = sadcs_b200.build_device(state["text"].data_ptr(), state["n"], state["sa"].data_ptr(),
                                          state["bwt"].data_ptr(), state["context"])
        return {"sa": state["sa"], "bwt": state["bwt"], "primary": primary}
    if op == "bwt":
        primary = sadcs_b200.build_device(state["text"].data_ptr(), state["n"], None, state["bwt"].data_ptr(),
                                          state["context"])
        return {"bwt": state["bwt"], "primary": primary}
    if op == "batch":
        primaries = sadcs_b200.build_batch_device(state["text"].data_ptr(), state["lengths"], state["sa"].data_ptr(),
                                                  state["bwt"].data_ptr(), state["context"])
        return {"sa": state["sa"], "bwt": state["bwt"], "primaries": np.asarray(primaries)}
    if op == "host":
        sa, bwt, primary = sadcs_b200.build(state["text"], context=state["context"], out_sa=state["sa"],
                                            out_bwt=state["bwt"])
        return {"sa": sa, "bwt": bwt, "primary": primary}
    if op == "serve":
        server, at = state["server"], state["at"]
        tickets = [server.submit(state["text"][a:b], sa=state["sa"][a:b], bwt=state["bwt"][a:b])
                   for a, b in zip(at, at[1:])]
        primaries = [server.wait(t)[2] for t in tickets]
        return {"sa": state["sa"], "bwt": state["bwt"], "primaries": np.asarray(primaries)}
    if op == "lcp":
        sadcs_b200.lcp_device(state["text"].data_ptr(), state["n"], state["sa"].data_ptr(), state["lcp"].data_ptr())
        return {"lcp": state["lcp"]}
    if op == "unbwt":
        sadcs_b200.inverse_bwt_device(state["bwt"].data_ptr(), state["n"], state["primary"], state["out"].data_ptr())
        return {"text": state["out"]}
    ok, index, _ = sadcs_b200.check_suffix_array_device(state["text"].data_ptr(), state["n"], state["sa"].data_ptr())
    primary = sadcs_b200.bwt_from_sa_device(state["text"].data_ptr(), state["n"], state["sa"].data_ptr(),
                                            state["bwt"].data_ptr())
    return {"ok": ok, "index": index, "bwt": state["bwt"], "primary": primary}


def work(case):
    """Bytes of the text read once and of the results written once; the work is on whole numbers."""
    op = case["op"]
    n = int(_lengths(case).sum()) if op in ("batch", "serve") else case["n"]
    per = {"build": 6, "host": 6, "batch": 6, "serve": 6, "bwt": 2, "lcp": 9, "unbwt": 2, "check": 6}[op]
    return {"bytes": per * n, "flops": 0}


def tolerance(case):
    return "exact"  # suffix arrays, BWTs, LCP arrays and texts are whole numbers


# ---- the results by other means ------------------------------------------------------------------

def _suffix_order(text):
    """The suffix array and every suffix's rank by prefix doubling with library sorts, 64-bit keys."""
    n = text.numel()
    key = torch.zeros(n, dtype=torch.int64, device="cuda")
    for k in range(7):  # seven characters, 1..256 each, 0 past the end
        key *= 257
        key[:max(0, n - k)] += text[k:].to(torch.int64) + 1
    h = 7
    while True:
        key, order = torch.sort(key)
        head = torch.ones(n, dtype=torch.int64, device="cuda")
        head[1:] = key[1:] != key[:-1]
        group = head.cumsum(0)
        rank = torch.empty_like(group)
        rank[order] = group
        if int(group[-1]) == n:
            return order, rank - 1
        key = rank * (n + 1)
        if h < n:
            key[:n - h] += rank[h:]
        h *= 2


def _lcp(text, order, rank):
    """Neighbours compared in growing steps: LCP lengths of unfinished pairs only."""
    n = text.numel()
    left, right = order[:-1].clone(), order[1:].clone()
    out = torch.zeros(n, dtype=torch.int64, device="cuda")
    open_ = torch.arange(1, n, device="cuda")
    while open_.numel():
        fits = (left < n) & (right < n)
        same = fits & (text[left.clamp(max=n - 1)] == text[right.clamp(max=n - 1)])
        out[open_[same]] += 1
        open_, left, right = open_[same], left[same] + 1, right[same] + 1
    return out


def exact(case, seed):
    op = case["op"]
    if op in ("batch", "serve") or case["n"] > 128 * MIB or (op == "lcp" and case["text"] != "uniform"):
        return None  # the last: comparing character by character would take too long on repeats
    text = _text(case["text"], case["n"], seed)
    if op == "unbwt":
        return {"text": text}
    order, rank = _suffix_order(text)
    if op == "lcp":
        return {"lcp": _lcp(text, order, rank)}
    row = int(rank[0])
    last = text[(order - 1).clamp_(min=0)]
    bwt = torch.cat([text[-1:], last[:row], last[row + 1:]])
    found = {"bwt": bwt, "primary": row + 1}
    if op == "check":
        found.update(ok=True, index=-1)
    elif op != "bwt":
        found["sa"] = order
    return found
