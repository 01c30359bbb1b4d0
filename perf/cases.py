"""What this library is timed on: searches as a program runs them.

A case is one pass of a searcher: a batch of records scored once from host
memory (`once`), a resident set scored again (`set`), a batch with its hits'
match starts through the matcher class (`match`), a text split into lines or
FASTQ records, scored and freed again (`lines`, `fastx`), many queries against
one set (`multi`), a burst of requests to the serving loop (`serve`).  Sizes
are those of the repository's workloads (24-byte line search, 300-residue
protein search, 50-1,000 nt query lists against reads, 1,000 nt against 10 kb -
1 Mb records, 20-2,000 residue serving mix), scaled so that a pass takes
microseconds to a fraction of a second.

Records, queries and texts are drawn on the GPU from the seed and kept in
pinned host memory, where a runner collects its batches; outputs go to pinned
buffers that the program keeps, or to the arrays the call returns.
"""
import math

import numpy as np
import torch

from ish_gb300 import native, workloads
from ish_gb300.matcher import StripedLocalMatcher, StripedSemiGlobalMatcher
from ish_gb300.scoring import KIND_NAMES, ScoringMatrix

MAX_CELLS = 3e11     # of a drawn case: no more than the largest listed one
MAX_RESIDUES = 2.4e8


def _case(how, matrix, algo, qlen, n, lengths, lo, hi, gaps, ends="FFTT", score=0.8, queries=1, name=None):
    c = dict(how=how, matrix=matrix, algo=algo, qlen=qlen, n=n, lengths=lengths, lo=lo, hi=hi, gap_open=gaps[0],
             gap_extend=gaps[1], ends=ends, score=score, queries=queries)
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # a short file searched for a word: 500 lines in one call
        _case("once", "ascii", "sg", 24, 500, "uniform", 20, 120, (3, 1), name="lines_500"),
        # one batch of the line runner: 100,000 lines from host memory
        _case("once", "ascii", "sg", 24, 100_000, "uniform", 20, 120, (3, 1), name="lines_100k"),
        # a text read whole: split into lines on the device, scored, match starts of the hits
        _case("lines", "ascii", "sg", 24, 300_000, "uniform", 0, 120, (3, 1), name="text_300k_lines"),
        # fuzzy text search with linear gaps (opening a gap costs no more than extending it)
        _case("once", "ascii", "sg", 31, 20_000, "uniform", 20, 120, (2, 2), score=0.7, name="lines_linear_gap"),
        # a small protein batch through the matcher class, local, with match starts
        _case("match", "blosum62", "local", 120, 3_000, "lognormal", 30, 5000, (10, 1), score=0.5,
              name="protein_batch_3k"),
        # a protein database kept on the device: 300-residue query, semi-global and local
        _case("set", "blosum62", "sg", 300, 400_000, "lognormal", 30, 5000, (10, 1), name="protein_sg_400k"),
        _case("set", "blosum62", "local", 300, 400_000, "lognormal", 30, 5000, (10, 1), name="protein_local_400k"),
        # a long protein against a smaller database
        _case("set", "blosum62", "local", 1501, 60_000, "lognormal", 30, 5000, (10, 1),
              name="protein_local_long_query"),
        # a query list against short reads in one batched launch
        _case("multi", "actgn", "sg", 1000, 90_000, "uniform", 100, 300, (3, 1), queries=32, name="reads_multi_32"),
        # sequencer output: FASTQ text split on the device, searched for an adapter, every end free
        _case("fastx", "actgn", "sg", 57, 250_000, "uniform", 100, 300, (3, 1), ends="TTTT", name="fastq_250k"),
        # a gene against chromosome-sized records
        _case("set", "actgn0", "sg", 1000, 1_000, "loguniform", 10_000, 1_000_000, (3, 1), name="long_records_1k"),
        # a burst of requests to a searcher that keeps its database on the device
        _case("serve", "blosum62", "mix", 2000, 60_000, "lognormal", 30, 5000, (10, 1), queries=12,
              name="serve_burst_12"),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _mean_length(c):
    if c["lengths"] == "uniform":
        return (c["lo"] + c["hi"]) / 2
    if c["lengths"] == "loguniform":
        return (c["hi"] - c["lo"]) / math.log(c["hi"] / c["lo"])
    return 420.0


def draw(rng):
    """One more case of the listed ones' ranges."""
    family = rng.choice(("once", "lines", "linear", "match", "protein", "multi", "fastx", "long", "serve"))
    any_ends = "FFTT" if rng.random() < 0.6 else "".join(rng.choice("FT") for _ in range(4))
    if family == "once":
        lo = rng.randrange(0, 40)
        c = _case("once", rng.choice(("ascii", "actgn")), rng.choice(("sg", "sg", "local")), _log(rng, 4, 100),
                  _log(rng, 100, 200_000), "uniform", lo, lo + rng.randrange(20, 200), (rng.randrange(2, 8), 1),
                  ends=any_ends)
    elif family == "lines":
        c = _case("lines", "ascii", rng.choice(("sg", "local")), _log(rng, 4, 60), _log(rng, 300, 400_000), "uniform",
                  0, rng.randrange(30, 250), (3, 1))
    elif family == "linear":
        g = rng.randrange(1, 4)
        c = _case("once", "ascii", rng.choice(("sg", "local")), _log(rng, 8, 100), _log(rng, 100, 20_000), "uniform",
                  20, rng.randrange(40, 150), (g, g), score=0.7)
    elif family == "match":
        c = _case("match", "blosum62", rng.choice(("sg", "local")), _log(rng, 20, 600), _log(rng, 100, 30_000),
                  "lognormal", 30, 5000, (rng.randrange(8, 13), rng.randrange(1, 3)), score=0.5)
    elif family == "protein":
        c = _case("set", "blosum62", rng.choice(("sg", "local")), _log(rng, 20, 2000), _log(rng, 2_000, 400_000),
                  "lognormal", 30, 5000, (rng.randrange(8, 13), rng.randrange(1, 3)), ends=any_ends)
    elif family == "multi":
        c = _case("multi", "actgn", "sg", _log(rng, 100, 1000), _log(rng, 2_000, 90_000), "uniform", 100, 300, (3, 1),
                  queries=_log(rng, 2, 48))
    elif family == "fastx":
        c = _case("fastx", "actgn", "sg", _log(rng, 12, 200), _log(rng, 500, 300_000), "uniform", 50,
                  rng.randrange(100, 400), (3, 1), ends=any_ends)
    elif family == "long":
        c = _case("set", "actgn0", rng.choice(("sg", "local")), _log(rng, 50, 1500), _log(rng, 10, 900), "loguniform",
                  10_000, 1_000_000, (3, 1))
    else:
        c = _case("serve", "blosum62", "mix", _log(rng, 200, 2000), _log(rng, 3_000, 60_000), "lognormal", 30, 5000,
                  (10, 1), queries=rng.randrange(2, 13))
    mean = max(_mean_length(c), 1.0)
    most = min(MAX_CELLS / (c["qlen"] * c["queries"]), MAX_RESIDUES) / mean
    c["n"] = max(4, min(c["n"], int(most)))
    return c


# ---- inputs ----

_P = {
    "actgn": [0.24875] * 4 + [0.005],
    "actgn0": [0.2985, 0.199, 0.199, 0.2985, 0.005],
    "blosum62": list(workloads.AA_BACKGROUND),
}


def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed) & 0x7FFFFFFFFFFF)
    return g


def _codes(g, n, matrix):
    """n i.i.d. residues: printable bytes, or the matrix's codes at its background frequencies."""
    if matrix == "ascii":
        return torch.randint(0x20, 0x7F, (n,), generator=g, device="cuda", dtype=torch.uint8)
    cdf = torch.tensor(np.cumsum(_P[matrix])[:-1], device="cuda", dtype=torch.float32)
    out = torch.empty(n, dtype=torch.uint8, device="cuda")
    for a in range(0, n, 1 << 26):
        b = min(n, a + (1 << 26))
        out[a:b] = torch.bucketize(torch.rand(b - a, generator=g, device="cuda"), cdf, out_int32=True).to(torch.uint8)
    return out


def _lengths(g, c):
    n, lo, hi = c["n"], c["lo"], c["hi"]
    if c["lengths"] == "uniform":
        return torch.randint(lo, hi + 1, (n,), generator=g, device="cuda")
    if c["lengths"] == "loguniform":
        u = torch.rand(n, generator=g, device="cuda", dtype=torch.float64)
        return torch.exp(math.log(lo) + u * math.log(hi / lo)).round().long()
    z = torch.randn(n, generator=g, device="cuda", dtype=torch.float64)
    return torch.exp(math.log(350.0) + 0.6 * z).round().long().clamp(lo, hi)


def _queries(g, c):
    """The case's query lengths and sequences: one of qlen residues, or a list up to qlen."""
    if c["queries"] == 1:
        sizes = [c["qlen"]]
    else:
        lo = max(20 if c["how"] == "serve" else 50, 1)
        lo = min(lo, c["qlen"])
        sizes = torch.randint(lo, c["qlen"] + 1, (c["queries"],), generator=g, device="cuda").tolist()
    return [_codes(g, s, c["matrix"]) for s in sizes]


def _records(g, c, queries):
    """Concatenated records and their n + 1 offsets (device); every hundredth holds a mutated copy of a query."""
    lens = _lengths(g, c)
    off = torch.zeros(c["n"] + 1, dtype=torch.int64, device="cuda")
    torch.cumsum(lens, 0, out=off[1:])
    recs = _codes(g, int(off[-1]), c["matrix"])
    pick = torch.arange(0, c["n"], 100, device="cuda") + torch.randint(0, 100, (1,), generator=g, device="cuda")
    pick = pick[pick < c["n"]]
    for k, q in enumerate(queries[:4]):
        w = pick[k::min(4, len(queries))]
        w = w[lens[w] >= len(q)]
        if len(w) == 0:
            continue
        at = off[w] + (torch.rand(len(w), generator=g, device="cuda") * (lens[w] - len(q) + 1)).long()
        copy = q.expand(len(w), -1).clone()
        sub = torch.rand(copy.shape, generator=g, device="cuda") < 0.08
        copy[sub] = _codes(g, int(sub.sum()), c["matrix"])
        recs[at[:, None] + torch.arange(len(q), device="cuda")] = copy
    return recs, off


def _host(t, dtype):
    """A pinned host array of t's values, as a runner's batch buffer."""
    a = torch.empty(max(t.numel(), 1), dtype=t.dtype, pin_memory=True)[: t.numel()]
    a.copy_(t)
    return a.numpy().view(dtype)


def _spread(recs, off, head, tail):
    """A text of '\\n' holding every record after `head` bytes and before `tail` bytes: (text, starts of the records)."""
    lens = off[1:] - off[:-1]
    size = lens + head + tail
    start = torch.cumsum(size, 0) - size + head
    text = torch.full((int(size.sum()),), 10, dtype=torch.uint8, device="cuda")
    at = torch.repeat_interleave(start - off[:-1], lens) + torch.arange(len(recs), device="cuda")
    text[at] = recs
    return text, start


def _text(g, c, recs, off):
    if c["how"] == "lines":
        return _spread(recs, off, 0, 1)[0]
    # FASTQ: "@r0000000\n" sequence "\n+\n" quality "\n"
    lens = off[1:] - off[:-1]
    letters = torch.tensor(list(b"ACGTN"), dtype=torch.uint8, device="cuda")
    head = 10
    qual = torch.randint(33, 74, (len(recs),), generator=g, device="cuda", dtype=torch.uint8)
    body = lens + head + 3 + lens + 1
    at0 = torch.cumsum(body, 0) - body
    text = torch.full((int(body.sum()),), 10, dtype=torch.uint8, device="cuda")
    idx = torch.arange(len(recs), device="cuda")
    text[torch.repeat_interleave(at0 + head - off[:-1], lens) + idx] = letters[recs.long()]
    text[torch.repeat_interleave(at0 + head + lens + 3 - off[:-1], lens) + idx] = qual
    text[at0] = ord("@")
    text[at0 + 1] = ord("r")
    num = torch.arange(c["n"], device="cuda")
    for d in range(7):
        text[at0 + 8 - d] = (num // 10**d % 10 + 48).to(torch.uint8)
    text[at0 + head + lens + 1] = ord("+")
    return text


_CTX = None


def _context():
    """The program's engine context: one for the process, kept."""
    global _CTX
    if _CTX is None:
        _CTX = native.Context(0)
    return _CTX


class State:
    """What a program holds between passes; gives its queries and set back when dropped."""

    def __init__(self, case):
        self.case = case
        self.ctx = native.Context(0) if case["how"] == "serve" else _context()
        self.qids, self.sid, self.matcher = [], None, None
        self.records = self.offsets = self.text = self.out = None
        self.lists = {}

    def __del__(self):
        try:
            if self.case["how"] == "serve":
                self.ctx.close()
                return
            if self.sid is not None:
                self.ctx.records_free(self.sid)
            for q in self.qids:
                self.ctx.free_query(q)
        except Exception:
            pass


def _algo_of(c, k):
    return c["algo"] if c["algo"] != "mix" else ("sg", "local")[k & 1]


def _ends_mask(ends):
    bits = (native.FREE_QUERY_START, native.FREE_QUERY_END, native.FREE_TARGET_START, native.FREE_TARGET_END)
    return sum(b for b, e in zip(bits, ends) if e == "T")


def _inputs(case, seed):
    g = _gen(seed)
    queries = _queries(g, case)
    recs, off = _records(g, case, queries)
    return g, queries, recs, off


def prepare(case, seed):
    s = State(case)
    g, queries, recs, off = _inputs(case, seed)
    kind = KIND_NAMES[case["matrix"]]
    m = ScoringMatrix(kind)
    how = case["how"]
    if how == "match":
        q = m.decode(queries[0].cpu().numpy())
        cls = StripedSemiGlobalMatcher if case["algo"] == "sg" else StripedLocalMatcher
        more = {"sg_ends_free": case["ends"]} if case["algo"] == "sg" else {}
        s.matcher = cls(q, case["score"], matrix_kind=case["matrix"], gap_open=case["gap_open"],
                        gap_extend=case["gap_extend"], context=s.ctx, **more)
        s.qids = [s.matcher.query_id]
    else:
        for k, q in enumerate(queries):
            q = q.cpu().numpy()
            algo = native.ALGO_SEMI_GLOBAL if _algo_of(case, k) == "sg" else native.ALGO_LOCAL
            s.qids.append(s.ctx.set_query(q, kind, m.values, algo, case["gap_open"], case["gap_extend"],
                                          _ends_mask(case["ends"]), int(m.values[q, q].astype(np.int64).sum()),
                                          case["score"]))
    if how in ("lines", "fastx"):
        s.text = _host(_text(g, case, recs, off), np.uint8)
        return s
    s.records, s.offsets = _host(recs, np.uint8), _host(off, np.uint64)
    if how in ("set", "multi", "serve"):
        s.sid = s.ctx.records_load(s.records, s.offsets)
    if how in ("once", "set"):
        n = case["n"]
        types = {"score": torch.int32, "qend": torch.int32, "tend": torch.int32, "hit": torch.uint8,
                 "hit_idx": torch.int32}
        s.out = {k: torch.empty(n, dtype=t, pin_memory=True).numpy() for k, t in types.items()}
        s.out["hit_idx"] = s.out["hit_idx"].view(np.uint32)
    if how == "serve":
        s.ctx.serve_start(s.sid)
    return s


def _kept(s, key, values, room):
    """A list of hits in an array of fixed size that the program keeps, -1 past its end."""
    buf, used = s.lists.get(key) or (np.full(room, -1, np.int64), 0)
    k = len(values)
    buf[:k] = values
    buf[k:used] = -1
    s.lists[key] = (buf, k)
    return buf


def run(s):
    c, ctx = s.case, s.ctx
    how, n = c["how"], c["n"]
    if how in ("once", "set"):
        r = ctx.score(s.qids[0], s.records, s.offsets, out=s.out) if how == "once" else \
            ctx.score_set(s.qids[0], s.sid, out=s.out)
        return dict(r, hit_idx=_kept(s, "hit_idx", r["hit_idx"], n))
    if how == "match":
        r = s.matcher.batch_match(s.records, s.offsets)
        return {"score": r.score, "qend": r.query_end, "tend": r.target_end, "hit": r.hit,
                "hit_idx": _kept(s, "hit_idx", r.hit_idx, n), "start": _kept(s, "start", r.hit_start, n)}
    if how == "multi":
        r = ctx.score_multi(s.qids, s.sid, want=("score", "tend", "hit_idx"))
        return {"score": r["score"], "tend": r["tend"], "hits": np.array([len(h) for h in r["hit_idx"]]),
                "hit_idx": _kept(s, "hit_idx", np.concatenate(r["hit_idx"]), n * c["queries"])}
    if how == "serve":
        tickets = [ctx.submit(q) for q in s.qids]
        out = []
        for k, t in enumerate(tickets):
            r = None
            while r is None:
                r = ctx.poll(t, wait_ms=1000)
            out.append([_kept(s, (k, f), r[f], n) for f in ("hit_idx", "score", "qend", "tend")])
        return out
    bounds = None
    if how == "lines":
        sid, _ = ctx.records_load_lines(s.text, KIND_NAMES[c["matrix"]])
    else:
        sid, _, bounds = ctx.records_load_fastx(s.text, KIND_NAMES[c["matrix"]])
    r = ctx.score_set(s.qids[0], sid)
    starts = ctx.match_starts(s.qids[0], sid, r["hit_idx"], r["tend"][r["hit_idx"]])
    ctx.records_free(sid)
    return {"score": r["score"], "qend": r["qend"], "tend": r["tend"], "hit": r["hit"],
            "hit_idx": _kept(s, "hit_idx", r["hit_idx"], n), "start": _kept(s, "start", starts, n), "bounds": bounds}


def work(case):
    """Every residue (or text byte) read once and 13 bytes written per record and query; nine integer operations per
    cell of the recurrence (two gap updates of two adds and a maximum, one match of an add and two maxima)."""
    mean = _mean_length(case)
    residues = case["n"] * mean
    qmean = case["qlen"] if case["queries"] == 1 else (case["qlen"] + 35) / 2
    text = {"lines": residues + case["n"], "fastx": 2 * residues + 14 * case["n"]}.get(case["how"], residues)
    return {"bytes": text + 13.0 * case["n"] * case["queries"], "flops": 9.0 * residues * qmean * case["queries"]}


# ---- plain 64-bit restatement ----

def _gotoh(c, algo, q, recs, off):
    """Scores, query ends and target ends of one query against all records: affine-gap alignment row by row over the
    records' residues, in 64-bit integers, records of a chunk side by side (longest first)."""
    M = torch.tensor(ScoringMatrix(KIND_NAMES[c["matrix"]]).values, device="cuda").long()
    O, X, Q, n = c["gap_open"], c["gap_extend"], len(q), c["n"]
    qs, qe, ts, te = (e == "T" for e in c["ends"])
    lens = off[1:] - off[:-1]
    order = torch.argsort(lens, descending=True, stable=True)
    score, qend, tend = (torch.zeros(n, dtype=torch.int64, device="cuda") for _ in range(3))
    col = torch.arange(Q + 1, device="cuda")
    prof = M[:, q.long()]
    step = max(1, (1 << 27) // (Q + 1))
    for a in range(0, n, step):
        ids = order[a:a + step]
        L, first = lens[ids], off[:-1][ids]
        m = len(ids)
        top = torch.zeros(Q + 1, dtype=torch.int64, device="cuda")
        if algo == "sg" and not qs:
            top[1:] = -O - X * (col[1:] - 1)
        H = top.repeat(m, 1)
        E = H[:, 1:] - O if algo == "sg" else torch.zeros(m, Q, dtype=torch.int64, device="cuda")
        best = torch.full((m,), 0 if algo == "local" else -(1 << 40), dtype=torch.int64, device="cuda")
        row, bcol = torch.full_like(best, -1), torch.zeros_like(best)
        alive = torch.bincount(L, minlength=int(L.max()) + 1).cpu().numpy()
        live = m - np.cumsum(alive)
        for i in range(int(L.max())):
            k = int(live[i])
            h, e = H[:k], E[:k]
            T = torch.maximum(h[:, :-1] + prof[recs[first[:k] + i].long()], e)
            left = 0 if (algo == "local" or ts) else -O - X * i
            if algo == "local":
                T.clamp_(min=0)
            G = torch.cat([torch.full((k, 1), left, dtype=torch.int64, device="cuda"), T], 1)
            F = torch.cummax(G + col * X, 1).values[:, :-1] - O - X * col[:-1]
            G[:, 1:] = torch.maximum(T, F)
            H[:k] = G
            E[:k] = torch.maximum(e - X, G[:, 1:] - O)
            if algo == "local":
                top_of, _ = G[:, 1:].max(1)
                up = top_of > best[:k]
                at = torch.where(G[:, 1:] == top_of[:, None], col[:-1], Q).amin(1)
                bcol[:k] = torch.where(up, at, bcol[:k])
            else:
                top_of = G[:, -1]
                up = top_of > best[:k]
            row[:k] = torch.where(up, i, row[:k])
            best[:k] = torch.where(up, top_of, best[:k])
        if algo == "local":
            s, r, b = best, row, bcol
        else:
            last = H[:, 1:]
            s, r = (best, row) if te else (torch.full_like(best, -(1 << 40)), L - 1)
            b = torch.full_like(best, Q - 1)
            if not te and not qe:
                s = last[:, -1]
            if qe:
                mx = last.max(1).values
                at = torch.where(last == mx[:, None], col[:-1], Q).amin(1)
                over, tie = mx > s, (mx == s) & (r == L - 1) & (at < b)
                s, r, b = torch.where(over, mx, s), torch.where(over, L - 1, r), torch.where(over | tie, at, b)
            empty = L == 0
            s, r, b = (torch.where(empty, 0, v) for v in (s, r, b))
        score[ids], tend[ids], qend[ids] = s, r, b
    return score, qend, tend


def _decide(c, algo, mx, s, qe, te):
    s32, m32, thr = s.float(), torch.tensor(float(mx), device="cuda"), torch.tensor(c["score"], device="cuda")
    if algo == "sg":
        return (s32 >= m32 * thr) & (s32 / m32 >= thr)
    return (s32 > thr * m32) & (te > 0) & (qe > 0) & (s32 / m32 >= thr)


def exact(case, seed):
    """Scores, ends and hits in plain 64-bit integers; None where rows would take too long one by one (long records),
    where results follow the lane order of the CPU passes (linear gaps), and for the serving burst."""
    if case["lengths"] == "loguniform" or case["gap_open"] <= case["gap_extend"] or case["how"] == "serve":
        return None
    g, queries, recs, off = _inputs(case, seed)
    if sum(len(q) for q in queries) * len(recs) > 8e10:
        return None
    values = ScoringMatrix(KIND_NAMES[case["matrix"]]).values

    def padded(v, room):
        return torch.cat([v, torch.full((room - len(v),), -1, dtype=torch.int64, device="cuda")])

    res = []
    for k, q in enumerate(queries):
        algo = _algo_of(case, k)
        s, qe, te = _gotoh(case, algo, q, recs, off)
        qh = q.cpu().numpy()
        res.append((s, qe, te, _decide(case, algo, int(values[qh, qh].astype(np.int64).sum()), s, qe, te)))
    if case["how"] == "multi":
        hits = [torch.nonzero(r[3])[:, 0] for r in res]
        return {"score": torch.stack([r[0] for r in res]).int(), "tend": torch.stack([r[2] for r in res]).int(),
                "hits": np.array([len(h) for h in hits]),
                "hit_idx": padded(torch.cat(hits), case["n"] * case["queries"])}
    s, qe, te, hit = res[0]
    out = {"score": s.int(), "qend": qe.int(), "tend": te.int(), "hit": hit.to(torch.uint8),
           "hit_idx": padded(torch.nonzero(hit)[:, 0], case["n"])}
    if case["how"] not in ("once", "set"):
        out["start"] = None
    if case["how"] in ("lines", "fastx"):
        out["bounds"] = None
    return out
