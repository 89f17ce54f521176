"""The work a user of this package has it do, as cases that can be timed one by one.

Every case goes through the public entry points with host queries in and host results out, as a
search tool or a read mapper calls them: plain scans of a resident database (best hit, every
target's score, every target's ends, every target's alignment), a batch of queries in all modes,
pairwise batches with and without the per-position maxima, and single pairs. Residues, lengths and
scorings follow the generators of the repository's benchmark: DNA +2/-1, and a protein matrix with a
positive diagonal, log-normal target lengths (median 300, sigma 0.8) and gaps 11/1. Databases and
scratches are built beforehand, as a program that searches one database many times keeps them.
"""
import math

import numpy as np
import torch

import hyalite_b200 as hy

HIT = np.dtype([("score", "<i4"), ("pad", "<u4"), ("db_index", "<u8"), ("query_end", "<i8"), ("target_end", "<i8")])
ALIGNMENT = np.dtype([("score", "<i4"), ("pad", "<u4"), ("query_start", "<u8"), ("query_end", "<u8"),
                      ("target_start", "<u8"), ("target_end", "<u8"), ("n_ops", "<u8"), ("ops_offset", "<u8")])
MODES = {"sw": hy.Mode.Sw, "nw": hy.Mode.Nw, "hw": hy.Mode.Hw, "shw": hy.Mode.Shw, "ov": hy.Mode.Ov}
BATCH_MODES = ("sw", "nw", "hw", "shw", "ov")
MEAN_PROTEIN = 300.0 * math.exp(0.8 * 0.8 / 2)  # mean target length of the protein generator
EXACT_CELL_STEPS = 3e10  # what exact() spends at most: values updated over all its steps


def _case(kind, **kw):
    c = {"kind": kind, "alphabet": "protein", "mode": "sw", "ends": True, "n": 1, "q": 100}
    c.update(kw)
    return c


def listed():
    return [
        # One adapter or probe against a small DNA library, best hit with its ends: launch latency.
        dict(_case("scan", alphabet="dna", n=10_000, q=64), name="scan_dna_small"),
        # One protein of typical length against a database, best hit with its ends: the plain search.
        dict(_case("scan", n=50_000, q=350), name="scan_protein_q350"),
        # A very long protein: many query passes, and targets whose scores need 32 bits.
        dict(_case("scan", n=50_000, q=5000), name="scan_protein_q5000"),
        # Every target's score and ends, for a report of all hits.
        dict(_case("scan_all", n=50_000, q=500), name="scan_all_protein_q500"),
        # Every read's score against one amplicon, the query aligned end to end (odd length).
        dict(_case("scan_scores", alphabet="reads", mode="hw", ends=False, n=200_000, q=731), name="scan_scores_reads_hw"),
        # A batch of queries of all lengths and modes against one set of reads.
        dict(_case("batch", alphabet="reads", n=100_000, q=25), name="batch_reads_all_modes"),
        # Reads against their candidate windows, semi-global: the mapper's inner loop.
        dict(_case("pairs", alphabet="reads", mode="hw", n=200_000, q=150), name="pairs_reads_hw"),
        # Protein pairs of ragged lengths, local: all queries differ.
        dict(_case("pairs", n=5_000, q=0), name="pairs_protein_sw"),
        # Mate rescue: the best score at every window position and the second-best peak.
        dict(_case("position_max", alphabet="reads", n=100_000, q=150), name="position_max_rescue"),
        # Every target's full alignment, for a result page or a multiple alignment.
        dict(_case("aligned", n=10_000, q=600), name="scan_all_aligned_q600"),
        # One pair with its alignment, and one pair's score and ends: interactive calls.
        dict(_case("align", q=2000), name="align_one_2000"),
        dict(_case("pair", q=2000), name="pair_one_2000"),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["scan", "scan", "scan_all", "scan_scores", "batch", "pairs", "pairs", "position_max",
                       "aligned", "align", "pair"])
    mode = rng.choice(["sw", "sw", "sw", "nw", "hw", "shw", "ov"])
    if kind in ("scan", "scan_all", "scan_scores"):
        alphabet = rng.choice(["dna", "protein", "protein", "reads"])
        return _case(kind, alphabet=alphabet, mode=mode, ends=kind == "scan_all" or (kind == "scan" and rng.random() < 0.75),
                     n=_log(rng, 1_000, 50_000), q=_log(rng, 30, 5000 if kind != "scan_all" else 1500))
    if kind == "batch":
        return _case(kind, alphabet="reads", n=_log(rng, 5_000, 100_000), q=_log(rng, 5, 25))
    if kind == "pairs":
        if rng.random() < 0.5:
            return _case(kind, mode=mode, ends=rng.random() < 0.7, n=_log(rng, 100, 5_000), q=0)
        return _case(kind, alphabet="reads", mode=mode, ends=rng.random() < 0.7, n=_log(rng, 1_000, 200_000),
                     q=rng.choice([75, 100, 101, 150, 151, 250]))
    if kind == "position_max":
        return _case(kind, alphabet="reads", n=_log(rng, 1_000, 100_000), q=rng.choice([75, 100, 101, 150, 151, 250]))
    if kind == "aligned":
        return _case(kind, alphabet=rng.choice(["dna", "protein"]), mode=mode, n=_log(rng, 100, 10_000), q=_log(rng, 50, 1000))
    return _case(kind, mode=mode, ends=kind == "pair" and rng.random() < 0.7, q=_log(rng, 100, 4000))


# ---- inputs ------------------------------------------------------------------------------------

def _scoring(case):
    if case["alphabet"] != "protein":
        go = 6 if case["kind"] in ("pairs", "position_max") else 2
        return hy.Scoring(4, [2 if a == b else -1 for a in range(4) for b in range(4)], go, 1)
    base = np.random.default_rng(12345)
    mat = base.integers(-4, 4, size=(20, 20))
    mat = np.triu(mat) + np.triu(mat, 1).T
    mat[np.diag_indices(20)] = base.integers(4, 12, size=20)
    return hy.Scoring(20, [int(v) for v in mat.reshape(-1)], 11, 1)


class _Draw:
    """Seeded residues and lengths, made on the GPU."""

    def __init__(self, case, seed):
        self.g = torch.Generator(device="cuda")
        self.g.manual_seed(seed)
        self.al = 20 if case["alphabet"] == "protein" else 4
        p = np.random.default_rng(54321).dirichlet(np.full(20, 4.0)) if self.al == 20 else np.full(4, 0.25)
        self.cdf = torch.tensor(np.cumsum(p)[:-1], dtype=torch.float32, device="cuda")

    def rand(self, *shape):
        return torch.rand(shape, generator=self.g, device="cuda")

    def ints(self, lo, hi, *shape):
        return torch.randint(lo, hi, shape, generator=self.g, device="cuda")

    def residues(self, n):
        return torch.searchsorted(self.cdf, self.rand(n)).to(torch.uint8)

    def protein_lengths(self, n):
        x = torch.randn((n,), generator=self.g, device="cuda")
        return torch.exp(math.log(300.0) + 0.8 * x).round().clamp(20, 35_000).long()

    def mutated(self, x, rate):
        """`x` with a share `rate` of its residues replaced."""
        return torch.where(self.rand(*x.shape) < rate, self.residues(x.numel()).view(x.shape), x)


def _offsets(lengths):
    off = torch.zeros(lengths.numel() + 1, dtype=torch.int64, device=lengths.device)
    off[1:] = torch.cumsum(lengths, 0)
    return off


def _reads(d, n, length, genome):
    """Reads of `length` from `genome`: 2% substitutions and, in three of four, one 1..3-base indel."""
    j = torch.arange(length, device="cuda")[None, :]
    start = d.ints(600, genome.numel() - 600 - length, n)
    at = d.ints(0, length, n)[:, None]
    size = d.ints(1, 4, n)[:, None]
    kind = d.rand(n)[:, None]
    shift = torch.where(kind < 0.375, (j >= at) * size, torch.where(kind < 0.75, -((j >= at) * torch.minimum(j - at, size)), 0))
    return d.mutated(genome[start[:, None] + j + shift], 0.02 * 4 / 3), start


def _database(case, d, query):
    """(residues, offsets) on the host; a half percent of the targets hold a mutated piece of the query."""
    n = case["n"]
    if case["alphabet"] == "reads":
        genome = d.residues(5_000_000)
        if query is not None:
            genome[1000: 1000 + query.numel()] = query
        reads, _ = _reads(d, n, 150, genome)
        off = torch.arange(n + 1, device="cuda") * 150
        return reads.reshape(-1).cpu().numpy(), off.cpu().numpy().astype(np.uint64)
    lengths = d.ints(50, 301, n) if case["alphabet"] == "dna" else d.protein_lengths(n)
    off = _offsets(lengths)
    res = d.residues(int(off[-1])).cpu().numpy()
    off = off.cpu().numpy()
    planted = d.mutated(query[None, :].expand(8, -1), 0.05 if case["alphabet"] == "dna" else 0.3).cpu().numpy()
    for i, k in enumerate(d.ints(0, n, max(1, n // 200)).tolist()):
        piece = planted[i % 8][: off[k + 1] - off[k]]
        res[off[k]: off[k] + len(piece)] = piece
    return res, off.astype(np.uint64)


def _pair(case, d):
    """A pair of related sequences of about the same length."""
    q = d.residues(case["q"])
    t = d.mutated(q, 0.15)
    cut = int(d.ints(0, case["q"] // 2, 1))
    return q.cpu().numpy(), torch.cat([t[:cut], d.residues(1 + case["q"] // 50), t[cut:]]).cpu().numpy()


def _pairs(case, d):
    """(query residues, offsets, target residues, offsets) on the host."""
    n = case["n"]
    if case["q"]:
        genome = d.residues(10_000_000)
        reads, start = _reads(d, n, case["q"], genome)
        # Every window length equally often, in a seeded order: the same number of residues for every seed.
        width = torch.linspace(max(200, case["q"] + 10), 500, n, device="cuda").long()[torch.argsort(d.rand(n))]
        first = start - (d.rand(n) * (width - case["q"])).long()
        t_off = _offsets(width)
        row = torch.repeat_interleave(torch.arange(n, device="cuda"), width)
        t = genome[first[row] + torch.arange(int(t_off[-1]), device="cuda") - t_off[row]]
        q, q_off = reads.reshape(-1), torch.arange(n + 1, device="cuda") * case["q"]
    else:
        ql, tl = d.protein_lengths(n).clamp(max=4000), d.protein_lengths(n).clamp(max=4000)
        q_off, t_off = _offsets(ql), _offsets(tl)
        q, t = d.residues(int(q_off[-1])), d.residues(int(t_off[-1]))
        row = torch.repeat_interleave(torch.arange(n, device="cuda"), tl)
        at = torch.arange(t.numel(), device="cuda") - t_off[row]
        t = torch.where(at < ql[row], d.mutated(q[(q_off[row] + at).clamp(max=q.numel() - 1)], 0.6), t)
    host = lambda x, dt: x.cpu().numpy().astype(dt)  # noqa: E731
    return host(q, np.uint8), host(q_off, np.uint64), host(t, np.uint8), host(t_off, np.uint64)


def _ops_room(case):
    """Bytes a program sets aside for the operations of a call's alignments."""
    return int(case["n"] * (case["q"] + 1.5 * (MEAN_PROTEIN if case["kind"] == "aligned" else case["q"]))) + 40_000


def _build(res, off, scoring, mode, search, max_query_len):
    return (hy.Database.builder().sequences_concat(res, off).scoring(scoring).mode(mode).search_type(search)
            .max_query_len(max_query_len).build())


def prepare(case, seed):
    d = _Draw(case, seed)
    s = {"case": case, "kind": case["kind"], "scoring": _scoring(case), "mode": MODES[case["mode"]],
         "search": hy.SearchType.ScoreEnd if case["ends"] else hy.SearchType.Score}
    if case["kind"] in ("align", "aligned"):
        s["ops"] = np.zeros(_ops_room(case), np.uint8)
    if case["kind"] in ("align", "pair"):
        s["query"], s["target"] = _pair(case, d)
    elif case["kind"] in ("pairs", "position_max"):
        s["pairs"] = _pairs(case, d)
        s["colmax"] = np.empty(int(s["pairs"][3][-1]), np.int32) if case["kind"] == "position_max" else None
    elif case["kind"] == "batch":
        n_q = case["q"]
        lengths = d.ints(32, 2001, n_q).tolist()
        queries = [d.residues(n).cpu().numpy() for n in lengths]
        res, off = _database(case, d, torch.from_numpy(queries[0]).cuda())
        s["dbs"] = [_build(res, off, s["scoring"], MODES[m], hy.SearchType.ScoreEnd, 2000) for m in BATCH_MODES]
        s["batch"] = hy.Batch(s["dbs"], max_queries=n_q)
        s["q_res"], s["q_off"] = hy.concat(queries)
        s["which"] = np.arange(n_q, dtype=np.uint32) % len(BATCH_MODES)
        s["batch"].tune(queries, s["which"])
    else:
        query = d.residues(case["q"])
        s["query"] = query.cpu().numpy()
        s["res"], s["off"] = _database(case, d, query)
        search = hy.SearchType.alignment(hy.USIZE_MAX) if case["kind"] == "aligned" else s["search"]
        s["db"] = _build(s["res"], s["off"], s["scoring"], s["mode"], search, case["q"])
        s["scratch"] = hy.Scratch(s["db"])
    return s


# ---- one pass ------------------------------------------------------------------------------------

def _hit(h):
    return {"score": h.score, "db_index": h.db_index, "query_end": -1 if h.query_end is None else h.query_end,
            "target_end": -1 if h.target_end is None else h.target_end}


def _fields(records, dtype, n, drop=("pad",)):
    a = np.frombuffer(records, dtype=dtype, count=n)
    return {f: a[f] for f in dtype.names if f not in drop}


def _kept(state, ops):
    """The operations in the program's own buffer, zeros after them."""
    state["ops"][: len(ops)] = ops
    state["ops"][len(ops): state.get("ops_end", 0)] = 0
    state["ops_end"] = len(ops)
    return state["ops"]


def run(state):
    kind = state["kind"]
    if kind == "scan":
        return _hit(state["db"].scan(state["scratch"], state["query"]))
    if kind == "scan_scores":
        return {"score": state["db"].scan_scores_array(state["scratch"], state["query"])}
    if kind == "scan_all":
        return _fields(state["db"].scan_all_array(state["scratch"], state["query"]), HIT, state["case"]["n"])
    if kind == "aligned":
        records, ops = state["db"].scan_all_aligned_arrays(state["scratch"], state["query"])
        return dict(_fields(records, ALIGNMENT, state["case"]["n"]), ops=_kept(state, ops))
    if kind == "batch":
        hits = state["batch"].scan_arrays(state["q_res"], state["q_off"], state["which"])
        return _fields(hits, HIT, state["case"]["q"])
    if kind == "pairs":
        hits, (err, _) = hy.align_pairs_arrays(*state["pairs"], state["scoring"], state["mode"], state["search"])
        if err is not None:
            raise err
        return _fields(hits, HIT, state["case"]["n"])
    if kind == "position_max":
        hits, colmax, second, (err, _) = hy.align_pairs_position_max_arrays(*state["pairs"], state["scoring"], 20,
                                                                            state["colmax"])
        if err is not None:
            raise err
        return dict(_fields(hits, HIT, state["case"]["n"]), colmax=colmax, second=second)
    if kind == "pair":
        return _hit(hy.align_pair(state["query"], state["target"], state["scoring"], state["mode"], state["search"]))
    a = hy.align(state["query"], state["target"], state["scoring"], state["mode"], hy.USIZE_MAX)
    return {"score": a.score, "query_start": a.query_start, "query_end": a.query_end, "target_start": a.target_start,
            "target_end": a.target_end, "ops": _kept(state, np.frombuffer(a.ops_bytes, np.uint8))}


# ---- what a pass cannot do without -----------------------------------------------------------------

OPS_PER_CELL = 8.0  # two gap updates (add, subtract, max each), the diagonal's add and the cell's max


def work(case):
    """Each residue read and each result written once; OPS_PER_CELL integer operations a cell."""
    kind, n, q = case["kind"], case["n"], case["q"]
    if kind in ("align", "pair"):
        return {"bytes": 2.0 * q + (2.0 * q if kind == "align" else 32.0), "flops": OPS_PER_CELL * q * q * 1.02}
    target = {"dna": 175.0, "reads": 150.0, "protein": MEAN_PROTEIN}[case["alphabet"]]
    if kind in ("pairs", "position_max"):
        if q:
            target = (max(200, q + 10) + 500) / 2
        query = q or MEAN_PROTEIN
        out = 32.0 + (4.0 * target + 8.0 if kind == "position_max" else 0.0)
        return {"bytes": n * (query + target + out), "flops": OPS_PER_CELL * n * query * target}
    if kind == "batch":
        return {"bytes": n * target + q * (1016.0 + 32.0), "flops": OPS_PER_CELL * n * target * q * 1016.0}
    out = {"scan": 32.0, "scan_scores": 4.0 * n, "scan_all": 32.0 * n, "aligned": n * (56.0 + target)}[kind]
    return {"bytes": n * target + q + out, "flops": OPS_PER_CELL * n * target * q}


# ---- the same scores in 64 bits ---------------------------------------------------------------------

def _gotoh_scores(q, t, t_len, scoring, mode):
    """Best scores of queries q [T, m] against targets t [T, n] of lengths t_len [T], 64-bit, swept by
    antidiagonals: cell (i, j) of diagonal k = i + j sits at index i."""
    T, m = q.shape
    al, go, ge = scoring.alphabet_len(), scoring.gap_open(), scoring.gap_ext()
    mat = torch.tensor(scoring.matrix(), dtype=torch.int64, device="cuda")
    top_free, left_free = mode in ("sw", "hw", "ov"), mode in ("sw", "ov", "shw")
    low = -(1 << 40)
    i = torch.arange(m + 1, device="cuda")
    full = lambda: torch.full((T, m + 1), low, dtype=torch.int64, device="cuda")  # noqa: E731
    h1, h2, e1, f1 = full(), full(), full(), full()
    best = torch.full((T,), low, dtype=torch.int64, device="cuda")
    qrow = torch.cat([torch.zeros((T, 1), dtype=torch.int64, device="cuda"), q.long()], 1) * al
    for k in range(m + int(t_len.max()) + 1):
        j = k - i
        e = torch.maximum(e1 - ge, h1 - go)
        f = full()
        f[:, 1:] = torch.maximum(f1[:, :-1] - ge, h1[:, :-1] - go)
        h = full()
        sub = mat[qrow + t[:, (j - 1).clamp(0, t.shape[1] - 1)].long()]
        h[:, 1:] = h2[:, :-1] + sub[:, 1:]
        h = torch.maximum(torch.maximum(h, e), f)
        h = h.clamp(min=0) if mode == "sw" else h
        if k <= m:
            h[:, k] = 0 if left_free or k == 0 else -(go + (k - 1) * ge)
            e[:, k] = f[:, k] = low
        h[:, 0] = 0 if top_free or k == 0 else -(go + (k - 1) * ge)
        e[:, 0] = f[:, 0] = low
        inside = (j >= 0) & (j <= t_len[:, None])
        h, e, f = (torch.where(inside, x, low) for x in (h, e, f))
        region = {"sw": inside, "nw": inside & (i == m) & (j == t_len[:, None]), "hw": inside & (i == m),
                  "shw": inside & (j == t_len[:, None])}.get(mode, inside & ((i == m) | (j == t_len[:, None])))
        best = torch.maximum(best, torch.where(region, h, low).amax(1))
        h2, h1, e1, f1 = h1, h, e, f
    return best


def _padded(res, off):
    length = torch.from_numpy(np.diff(off.astype(np.int64))).cuda()
    at = torch.from_numpy(off[:-1].astype(np.int64)).cuda()[:, None] + torch.arange(int(length.max()), device="cuda")
    return torch.from_numpy(res).cuda()[at.clamp(max=len(res) - 1)], length


def exact(case, seed):
    kind, q = case["kind"], case["q"]
    if kind == "batch" or (kind == "pairs" and not q):
        return None
    s = prepare(case, seed)
    if kind in ("align", "pair"):
        query, target = torch.from_numpy(s["query"].copy()).cuda()[None], torch.from_numpy(s["target"].copy()).cuda()[None]
        score = int(_gotoh_scores(query, target, torch.tensor([target.shape[1]], device="cuda"), s["scoring"], case["mode"]))
        if kind == "pair":
            return {"score": score, "db_index": 0, "query_end": None, "target_end": None}
        return {"score": score, "query_start": None, "query_end": None, "target_start": None, "target_end": None, "ops": None}
    if kind in ("pairs", "position_max"):
        res, off, query = s["pairs"][2], s["pairs"][3], torch.from_numpy(s["pairs"][0]).cuda().view(case["n"], q)
    else:
        res, off, query = s["res"], s["off"], torch.from_numpy(s["query"].copy()).cuda()[None].expand(case["n"], -1)
    longest = int(np.diff(off.astype(np.int64)).max())
    if float(case["n"]) * (q + 1) * (q + longest) > EXACT_CELL_STEPS:
        return None
    targets, length = _padded(res, off)
    score = torch.cat([_gotoh_scores(query[a: a + 20_000], targets[a: a + 20_000], length[a: a + 20_000], s["scoring"], case["mode"])
                       for a in range(0, case["n"], 20_000)]).cpu().numpy().astype(np.int32)
    if kind == "scan":
        return {"score": int(score.max()), "db_index": int(score.argmax()), "query_end": None, "target_end": None}
    if kind == "scan_scores":
        return {"score": score}
    if kind == "aligned":
        return {"score": score, **{f: None for f in ALIGNMENT.names if f not in ("score", "pad")}, "ops": None}
    out = {"score": score, "db_index": np.arange(case["n"]) if kind == "pairs" else None, "query_end": None, "target_end": None}
    if kind == "scan_all":
        out["db_index"] = np.arange(case["n"])
    if kind == "position_max":
        out["colmax"] = out["second"] = None
    return out
