"""The alignment work that performance is measured on.

Every case is one call of a program that holds a driver (SmithWatermanB200 or
Aligner: one engine, its scoring set) and gets new records for each call, as
the command line and the serving programs do: packed record sets go to the
engine, the whole path runs (score sweep, starting points, traceback walk, hit
order, strings) and the hits, or the pair maxima of a score-only call, come
back in host memory.  The records are host data by the path's nature.

  listed()            the cases
  draw(rng)           another case of the same ranges
  prepare(case, seed) the records (from the seed) and the driver kept for the case
  run(state)          one call; hits and strings as bytes in the program's own
                      buffers, maxima as floats
  exact(case, seed)   pair maxima in 64 bits, without the engine
  work(case)          what a call cannot do without

Five kinds of work:

  reads     DNA reads against adapters and their reverse complements, linear
            or affine gap (adapter search and trimming; 1 to 500,000 reads)
  proteins  protein queries against protein targets, linear or affine gap, hits,
            TXT records or only the matrix of maxima (batches, panels,
            all-against-all matrices)
  database  protein queries against a database that stays on the device
            (searches: one query's maxima, or the hits of a few queries)
  pairs     listed pairs of long sequences (genome fragments with their
            reverse complements, long proteins)
  genome    one long DNA query against one target and its reverse complement,
            all against all
"""
import math

import numpy as np
import torch

from pypaswas_b200 import programs, readers, scores, smith_waterman, workloads

DNA = workloads.DNA
AMINO = workloads.AMINO
AMINO_P = workloads.AMINO_FREQ
_COMP = np.zeros(256, dtype=np.uint8)
_COMP[np.frombuffer(b"ACGT", dtype=np.uint8)] = np.frombuffer(b"TGCA", dtype=np.uint8)


def listed():
    return [
        # one read arriving by itself (an interactive or streaming caller): launches and host steps only
        dict(name="one_read", kind="reads", reads=1, read_min=150, read_max=150, adapters=24, adapter_min=20,
             adapter_max=40, match=1.0, mismatch=-3.0, gap=-5.0, ext=0.0, minimum=8.0, out="hits"),
        # the adapter search of the benchmark's first configuration
        dict(name="reads_1k", kind="reads", reads=1000, read_min=150, read_max=150, adapters=50, adapter_min=30,
             adapter_max=60, match=1.0, mismatch=-3.0, gap=-5.0, ext=0.0, minimum=15.0, out="hits"),
        # the trimmer: a lane's worth of reads, records without strings, as Trimmer.trimmed_fasta takes them
        dict(name="trim_500k", kind="reads", reads=500_000, read_min=150, read_max=150, adapters=24, adapter_min=20,
             adapter_max=40, match=1.0, mismatch=-3.0, gap=-5.0, ext=0.0, minimum=8.0, out="records"),
        # scores that are no whole numbers (fp32 lanes), ragged reads, maxima and hits
        dict(name="reads_fractional", kind="reads", reads=3001, read_min=71, read_max=251, adapters=17, adapter_min=20,
             adapter_max=75, match=1.5, mismatch=-2.25, gap=-3.5, ext=0.0, minimum=15.0, out="both"),
        # the reference's own timing runs: 8 proteins against up to 340 targets, BLOSUM80, linear gap, TXT output
        dict(name="panel_txt", kind="proteins", queries=8, targets=340, median=350, q_max=1000, t_min=50, t_max=2000,
             matrix="BLOSUM80", gap=-5.0, ext=0.0, minimum=30.0, out="text"),
        # the headline batch: 400,000 pairs, affine gap, full path
        dict(name="batch_affine", kind="proteins", queries=200, targets=2000, median=350, q_max=1000, t_min=50,
             t_max=2000, matrix="BLOSUM62", gap=-11.0, ext=-1.0, minimum=30.0, out="hits"),
        # an all-against-all matrix of maxima (clustering, guide trees), linear gap
        dict(name="matrix_linear", kind="proteins", queries=701, targets=701, median=350, q_max=1000, t_min=50,
             t_max=2000, matrix="BLOSUM62", gap=-8.0, ext=0.0, minimum=30.0, out="maxima"),
        # one query's maxima over a resident database (a top-k request of the serving loop)
        dict(name="database_one", kind="database", queries=1, targets=50_000, median=350, q_max=1000,
             matrix="BLOSUM62", gap=-11.0, ext=-1.0, minimum=30.0, out="maxima"),
        # a serving batch of traceback requests
        dict(name="database_hits", kind="database", queries=6, targets=50_000, median=300, q_max=1000,
             matrix="BLOSUM62", gap=-11.0, ext=-1.0, minimum=30.0, out="hits"),
        # long DNA pairs, each with the target's reverse complement (the benchmark's third configuration)
        dict(name="long_pairs", kind="pairs", residues="dna", pairs=64, len_min=10_000, len_max=50_000, match=1.0,
             mismatch=-3.0, gap=-5.0, ext=0.0, minimum=100.0, factor=0.01, out="hits"),
        # one pair of genome fragments: the wavefront of a single pair
        dict(name="genome_pair", kind="genome", residues="dna", pairs=1, len_min=30_000, len_max=30_000, match=1.0,
             mismatch=-3.0, gap=-5.0, ext=0.0, minimum=100.0, factor=0.01, out="hits"),
        # long proteins, listed pairs, affine gap
        dict(name="long_proteins", kind="pairs", residues="protein", pairs=12, len_min=2000, len_max=8000,
             matrix="BLOSUM62", gap=-11.0, ext=-1.0, minimum=100.0, factor=0.01, out="hits"),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["reads", "reads", "proteins", "proteins", "database", "pairs", "genome"])
    if kind == "reads":
        fractional = rng.random() < 0.2
        n = _log(rng, 1, 30_000 if fractional else 400_000)
        a = rng.randint(36, 200)
        b = a if rng.random() < 0.4 else min(300, a + rng.randint(1, 100))
        lo = rng.randint(18, 40)
        adapters = rng.randint(1, 30)
        adapter_max = lo + rng.randint(0, 30)
        if n > 100_000:
            adapters, adapter_max = min(adapters, 16), min(adapter_max, 45)
        affine = rng.random() < 0.25
        if fractional:
            m = dict(match=1.5, mismatch=-2.25, gap=-3.5)
        else:
            m = rng.choice([dict(match=1.0, mismatch=-3.0, gap=-5.0), dict(match=5.0, mismatch=-3.0, gap=-5.0),
                            dict(match=2.0, mismatch=-2.0, gap=-3.0)])
        minimum = (15.0 if n < 20_000 else 12.0) * m["match"]
        return dict(kind="reads", reads=n, read_min=a, read_max=b, adapters=adapters, adapter_min=lo,
                    adapter_max=adapter_max, ext=-1.0 if affine else 0.0, minimum=minimum,
                    out=rng.choice(["hits", "records", "both"]), **m)
    protein = rng.choice([dict(matrix="BLOSUM62", gap=-11.0, ext=-1.0), dict(matrix="BLOSUM62", gap=-10.0, ext=-2.0),
                          dict(matrix="BLOSUM80", gap=-5.0, ext=0.0), dict(matrix="BLOSUM62", gap=-8.0, ext=0.0)])
    if kind == "proteins":
        t_min = rng.randint(60, 200)
        minimum = 60.0 if protein["gap"] == -5.0 else 45.0
        return dict(kind="proteins", queries=_log(rng, 1, 180), targets=_log(rng, 1, 1800),
                    median=rng.randint(150, 350), q_max=1000, t_min=t_min, t_max=t_min + _log(rng, 10, 1700),
                    minimum=minimum, factor=0.2 if protein["gap"] == -5.0 else 0.1,
                    out=rng.choice(["hits", "maxima", "both", "text"]), **protein)
    if kind == "database":
        return dict(kind="database", queries=rng.randint(1, 8), targets=_log(rng, 8000, 50_000),
                    median=rng.randint(80, 350), q_max=1000, minimum=60.0, out=rng.choice(["maxima", "hits"]),
                    **protein)
    if kind == "genome":
        n = _log(rng, 5000, 40_000)
        return dict(kind="genome", residues="dna", pairs=1, len_min=max(4500, n - rng.randint(0, n // 3)), len_max=n,
                    match=1.0, mismatch=-3.0, gap=-5.0, ext=0.0, minimum=100.0, factor=0.01, out="hits")
    if rng.random() < 0.5:
        hi = _log(rng, 4000, 40_000)
        return dict(kind="pairs", residues="dna", pairs=_log(rng, 1, 40), len_min=rng.randint(2500, hi), len_max=hi,
                    match=1.0, mismatch=-3.0, gap=-5.0, ext=0.0, minimum=100.0, factor=0.01, out="hits")
    hi = _log(rng, 1000, 8000)
    return dict(kind="pairs", residues="protein", pairs=_log(rng, 1, 24), len_min=rng.randint(700, hi), len_max=hi,
                minimum=100.0, factor=0.01, out="hits", **protein)


# ------------------------------------------------------------------ records
def _record_set(seqs, prefix):
    """Packed records, longest first (stable), as the reader's sort leaves them."""
    order = sorted(range(len(seqs)), key=lambda i: -len(seqs[i][1]))
    seqs = [seqs[i] for i in order]
    off = np.zeros(len(seqs) + 1, dtype=np.int64)
    np.cumsum([len(s) for _, s in seqs], out=off[1:])
    ids = [(prefix + str(i)).encode() for i, _ in seqs]
    id_off = np.zeros(len(seqs) + 1, dtype=np.int64)
    np.cumsum([len(i) for i in ids], out=id_off[1:])
    res = np.concatenate([s for _, s in seqs]) if seqs else np.zeros(0, np.uint8)
    return readers.RecordSet(np.ascontiguousarray(res), off, np.frombuffer(b"".join(ids), dtype=np.uint8), id_off)


def _random(rng, n, alphabet, p=None):
    return alphabet[rng.choice(len(alphabet), size=int(n), p=p)]


def _mutate(rng, a, alphabet, subs, indels=0.0):
    """Substitutions, then single-residue deletions and insertions."""
    a = a.copy()
    m = rng.random(len(a)) < subs
    a[m] = alphabet[rng.integers(0, len(alphabet), int(m.sum()))]
    if indels > 0:
        times = np.ones(len(a), dtype=np.int64)
        r = rng.random(len(a))
        times[r < indels / 2] = 0
        times[r > 1 - indels / 2] = 2
        a = np.repeat(a, times)
    return a


def _revcomp(a):
    return _COMP[a][::-1]


def _lengths(rng, n, median, hi, lo=100):
    return np.clip(np.round(rng.lognormal(np.log(median), 0.5, n)), min(lo, hi), hi).astype(np.int64)


def _reads(case, rng):
    """Uniform ACGT reads; 40% end in a prefix (8 residues and more) of an
    adapter with up to three substitutions.  Targets: adapters and their
    reverse complements."""
    n = case["reads"]
    adapters = [_random(rng, rng.integers(case["adapter_min"], case["adapter_max"] + 1), DNA)
                for _ in range(case["adapters"])]
    lens = rng.integers(case["read_min"], case["read_max"] + 1, n)
    lens = -np.sort(-lens)
    off = np.zeros(n + 1, dtype=np.int64)
    np.cumsum(lens, out=off[1:])
    res = DNA[rng.integers(0, 4, int(off[-1]), dtype=np.uint8)]
    carry = np.nonzero(rng.random(n) < 0.4)[0] if n > 1 else np.arange(n)
    which = rng.integers(0, len(adapters), len(carry))
    alen = np.array([len(a) for a in adapters])
    amat = np.zeros((len(adapters), int(alen.max())), dtype=np.uint8)
    for i, a in enumerate(adapters):
        amat[i, :len(a)] = a
    frag = np.minimum(rng.integers(8, int(alen.max()) + 1, len(carry)), np.minimum(alen[which], lens[carry]))
    cols = np.arange(amat.shape[1])
    inside = cols[None, :] < frag[:, None]
    at = (off[carry + 1] - frag)[:, None] + cols[None, :]
    res[at[inside]] = amat[which][inside]
    for k in range(3):
        some = rng.random(len(carry)) < 0.6 - 0.2 * k
        pos = off[carry + 1] - 1 - (rng.random(len(carry)) * frag).astype(np.int64)
        res[pos[some]] = DNA[rng.integers(0, 4, int(some.sum()))]
    width = len(str(max(n - 1, 1)))
    digits = (np.arange(n)[:, None] // 10 ** np.arange(width - 1, -1, -1)[None, :]) % 10 + 48
    ids = np.concatenate([np.full((n, 1), ord("r"), np.uint8), digits.astype(np.uint8)], axis=1)
    queries = readers.RecordSet(res, off, ids.reshape(-1), np.arange(n + 1, dtype=np.int64) * (width + 1))
    targets = [(str(i), a) for i, a in enumerate(adapters)]
    targets += [("%d_RC" % i, _revcomp(a)) for i, a in enumerate(adapters)]
    return queries, _record_set(targets, "adapter"), None


def _proteins(case, rng):
    """Background residue frequencies; a 150-residue domain (or what of it fits)
    in a third of the queries and, at 40% identity, in a third of the targets;
    the first query and, at 70%, the first target always carry it."""
    qlen = _lengths(rng, case["queries"], case["median"], case["q_max"])
    tlen = rng.integers(case["t_min"], case["t_max"] + 1, case["targets"])
    domain = _random(rng, 150, AMINO, AMINO_P)

    def one(n, d):
        s = _random(rng, n, AMINO, AMINO_P)
        if d is not None:
            d = d[:n]
            p = int(rng.integers(0, n - len(d) + 1))
            s[p:p + len(d)] = d
        return s

    q = [(i, one(n, domain if i == 0 or rng.random() < 0.32 else None)) for i, n in enumerate(qlen)]
    t = [(i, one(n, _mutate(rng, domain, AMINO, 0.6 if i else 0.3) if i == 0 or rng.random() < 0.32 else None))
         for i, n in enumerate(tlen)]
    return _record_set(q, "query"), _record_set(t, "target"), None


def _database(case):
    """The resident database: part of what the program keeps, the same for every call."""
    rng = np.random.default_rng(case["targets"])
    lens = _lengths(rng, case["targets"], 300, 1500, 50)
    flat = _random(rng, lens.sum(), AMINO, AMINO_P)
    cut = np.concatenate([[0], np.cumsum(lens)])
    return _record_set([(i, flat[cut[i]:cut[i + 1]]) for i in range(len(lens))], "db")


def _database_queries(case, rng, db):
    """Queries of which every second one holds a mutated stretch of a database sequence."""
    out = []
    for i, n in enumerate(_lengths(rng, case["queries"], case["median"], case["q_max"], 20)):
        s = _random(rng, n, AMINO, AMINO_P)
        if i % 2 == 0:
            k = int(rng.integers(0, len(db)))
            a = db.residues[db.offsets[k]:db.offsets[k + 1]][:n // 2]
            a = _mutate(rng, a, AMINO, 0.3)
            s[n // 4:n // 4 + len(a)] = a
        out.append((i, s))
    return _record_set(out, "request")


def _long(case, rng):
    """Pairs that share one homologous region (a fifth to a half of the shorter
    sequence, 85% identity, 2% indels); DNA targets come with their reverse
    complements, query i paired with targets i and i + pairs."""
    dna = case["residues"] == "dna"
    alphabet, p = (DNA, None) if dna else (AMINO, AMINO_P)
    n = case["pairs"]
    q, t = [], []
    for i in range(n):
        lq, lt = (int(v) for v in rng.integers(case["len_min"], case["len_max"] + 1, 2))
        a, b = _random(rng, lq, alphabet, p), _random(rng, lt, alphabet, p)
        ls = int(min(lq, lt) * rng.uniform(0.2, 0.5))
        pq, pt = int(rng.integers(0, lq - ls + 1)), int(rng.integers(0, lt - ls + 1))
        hom = _mutate(rng, a[pq:pq + ls], alphabet, 0.15, 0.02)[:lt - pt]
        b[pt:pt + len(hom)] = hom
        q.append(a)
        t.append(b)
    if dna:
        t = t + [_revcomp(b) for b in t]
    # records in the given order: the pair list names them
    sets = []
    for seqs, prefix in ((q, b"long"), (t, b"ref")):
        off = np.zeros(len(seqs) + 1, dtype=np.int64)
        np.cumsum([len(s) for s in seqs], out=off[1:])
        ids = [prefix + str(i).encode() for i in range(len(seqs))]
        id_off = np.zeros(len(seqs) + 1, dtype=np.int64)
        np.cumsum([len(i) for i in ids], out=id_off[1:])
        sets.append(readers.RecordSet(np.concatenate(seqs), off, np.frombuffer(b"".join(ids), dtype=np.uint8), id_off))
    pairs = [(i, i) for i in range(n)] + ([(i, i + n) for i in range(n)] if dna else [])
    return sets[0], sets[1], (pairs if case["kind"] == "pairs" else None)


def _records(case, seed):
    rng = np.random.default_rng([int(seed), 1])
    if case["kind"] == "reads":
        return _reads(case, rng)
    if case["kind"] == "proteins":
        return _proteins(case, rng)
    return _long(case, rng)


# ------------------------------------------------------------------- driver
def _settings(case):
    kw = dict(gap_score="%g" % case["gap"], gap_extension="%g" % case["ext"], minimum_score="%g" % case["minimum"],
              lower_limit_score="1.0", filter_factor="%g" % case.get("factor", 0.2), relative_score="0",
              base_score="0", query_identity="0", query_coverage="0")
    if "matrix" in case:
        kw["matrix_name"] = case["matrix"]
    else:
        kw.update(matrix_name="DNA-RNA", match_score="%g" % case["match"], mismatch_score="%g" % case["mismatch"],
                  any_score="1")
    return workloads.Settings(**kw)


_kept = {}  # the one driver a program keeps (by its scoring and, for a database, the database)


def _driver(case):
    key = tuple(sorted((k, v) for k, v in case.items() if k != "name"))
    if key not in _kept:
        for old in _kept.values():
            old["aligner"].smith_waterman.close()
        _kept.clear()
        st = _settings(case)
        kept = {"aligner": programs.Aligner(None, scores.make_score(st), st)}
        if case["kind"] == "database":
            kept["db"] = _database(case)
            engine = kept["aligner"].smith_waterman.engine
            engine.set_targets_packed(kept["db"].residues, kept["db"].offsets, np.arange(len(kept["db"])))
        _kept[key] = kept
    return _kept[key]


def prepare(case, seed):
    kept = _driver(case)
    if case["kind"] == "database":
        queries = _database_queries(case, np.random.default_rng([int(seed), 1]), kept["db"])
        return dict(kept, out=case["out"], queries=queries, targets=None, pairs=None)
    queries, targets, pairs = _records(case, seed)
    return dict(kept, out=case["out"], queries=queries, targets=targets, pairs=pairs)


def _capacity(case):
    """(hits, bytes of strings or text) that a call's own buffers hold, well above what these records give."""
    q, t, pairs, _ = _sizes(case)
    if case["kind"] == "reads":
        n = int(case["reads"] * (5 if case["minimum"] < 10 * case["match"] else 3)) + 512
        return n, n * 3 * (case["adapter_max"] + 20) + n * (160 if case["out"] == "text" else 0)
    if case["kind"] in ("proteins", "database"):
        n = pairs // 3 + 4096
        return n, n * 600 + 2_000_000
    return 16 * pairs + 64, pairs * 6 * case["len_max"] + 4096


def _into(buffer, data):
    """The bytes in the program's own buffer (zero past them), which is returned whole."""
    if len(data) > len(buffer):
        raise ValueError("%d bytes for a buffer of %d" % (len(data), len(buffer)))
    buffer[:len(data)] = data
    return buffer


def prepare(case, seed):
    kept = _driver(case)
    hits, text = _capacity(case)
    state = dict(kept, out=case["out"], targets=None, pairs=None)
    if case["out"] == "text":
        state["text"] = np.zeros(text, dtype=np.uint8)
    elif case["out"] != "maxima":
        state["hits"] = np.zeros(hits * 48, dtype=np.uint8)
        state["strings"] = np.zeros(text if case["out"] != "records" else 0, dtype=np.uint8)
    if case["kind"] == "database":
        state["queries"] = _database_queries(case, np.random.default_rng([int(seed), 1]), kept["db"])
    else:
        state["queries"], state["targets"], state["pairs"] = _records(case, seed)
    return state


def run(state):
    out, queries, targets, pairs = state["out"], state["queries"], state["targets"], state["pairs"]
    engine = state["aligner"].smith_waterman.engine
    if out == "text":
        text = state["aligner"].txt(queries, targets)
        return {"text": _into(state["text"], np.frombuffer(text.encode("ascii"), dtype=np.uint8))}
    if targets is None:  # the resident database
        engine.set_queries_packed(queries.residues, queries.offsets, np.arange(len(queries)) + engine.n_targets)
    else:
        qk, tk = smith_waterman.packed_id_keys(queries, targets)
        engine.set_queries_packed(queries.residues, queries.offsets, qk)
        engine.set_targets_packed(targets.residues, targets.offsets, tk)
    if out == "maxima":
        engine.align(score_only=True)
        return {"maxima": engine.pair_max()}
    if pairs is not None:
        engine.set_pairs([p[0] for p in pairs], [p[1] for p in pairs])
    engine.align()
    hits, strings = engine.hits_view()
    got = {"hits": _into(state["hits"], hits.view(np.uint8))}
    if out != "records":
        got["strings"] = _into(state["strings"], np.frombuffer(strings, dtype=np.uint8))
    if out == "both":
        got["maxima"] = engine.pair_max()
    return got


# ------------------------------------------------------------- work, exact
def _sizes(case):
    """(query residues, target residues, pairs, cells) of a call, in the mean."""
    if case["kind"] == "reads":
        q = case["reads"] * (case["read_min"] + case["read_max"]) / 2
        t = 2 * case["adapters"] * (case["adapter_min"] + case["adapter_max"]) / 2
        return q, t, case["reads"] * 2 * case["adapters"], q * t
    if case["kind"] == "proteins":
        q = case["queries"] * case["median"] * 1.1
        t = case["targets"] * (case["t_min"] + case["t_max"]) / 2
        return q, t, case["queries"] * case["targets"], q * t
    if case["kind"] == "database":
        q = case["queries"] * case["median"] * 1.1
        t = case["targets"] * 340.0
        return q, t, case["queries"] * case["targets"], q * t
    mean = (case["len_min"] + case["len_max"]) / 2
    n, both = case["pairs"], 2 if case["residues"] == "dna" else 1
    return n * mean, both * n * mean, both * n, both * n * mean * mean


def work(case):
    """Residues in and maxima or (at least) nothing out; per cell the adds and
    maxima of the score recurrence (5 linear, 10 affine)."""
    q, t, pairs, cells = _sizes(case)
    maxima = 4.0 * pairs if case["out"] in ("maxima", "both") else 0.0
    return {"bytes": q + (0.0 if case["kind"] == "database" else t) + maxima,
            "flops": cells * (10.0 if case["ext"] != 0.0 else 5.0)}


def _padded(rs, dim_code):
    """Records as a matrix of matrix indices, -1 past their ends."""
    lens = np.diff(rs.offsets)
    out = np.full((len(lens), max(1, int(lens.max()))), -1, dtype=np.int64)
    for i, n in enumerate(lens):
        out[i, :n] = rs.residues[rs.offsets[i]:rs.offsets[i + 1]].astype(np.int64) - dim_code
    return out, lens


def _maxima64(case, queries, targets):
    """Pair maxima in 64 bits: the recurrence over whole anti-diagonals, many
    pairs at a time (H = max(0, diagonal + s, left + gap, up + gap); affine:
    M = max(0, best(diagonal) + s), gap chains opened from M, best = max(M, X, Y))."""
    st = _settings(case)
    score = scores.make_score(st)
    gap, ext, affine, _, _ = scores.kernel_constants(score)
    code = scores.char_offset_code(score)
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    mat = np.asarray(scores.matrix_array(score), dtype=np.float64)
    neg = -1e300
    mat = torch.tensor(np.pad(mat, ((0, 1), (0, 1)), constant_values=-1e6), device=dev)  # index -1: past an end
    q, ql = _padded(queries, code)
    t, tl = _padded(targets, code)
    out = np.zeros((len(ql), len(tl)))
    step = max(256, 100_000 // min(len(ql), 512))
    for t0 in range(0, len(tl), step):  # records come longest first: blocks of like lengths
        lt = int(tl[t0:t0 + step].max())
        for q0 in range(0, len(ql), 512):
            lq = int(ql[q0:q0 + 512].max())
            qq = torch.tensor(q[q0:q0 + 512, :lq], device=dev)
            tt = torch.tensor(t[t0:t0 + step, :lt], device=dev)
            b = (len(qq), len(tt))
            width = min(lq, lt)
            swap = lt < lq  # the shorter sequence runs along the diagonal
            z = torch.zeros(b + (width + 1,), dtype=torch.float64, device=dev)
            best2, best1, m1 = z.clone(), z.clone(), z.clone()
            x1, y1 = torch.full_like(z, neg), torch.full_like(z, neg)
            top = torch.zeros(b, dtype=torch.float64, device=dev)
            short, long_ = (tt, qq) if swap else (qq, tt)
            rest = max(lq, lt)
            for d in range(lq + lt - 1):  # cells (i, d - i): i along the shorter one
                i0, i1 = max(0, d - rest + 1), min(width, d + 1)
                i = torch.arange(i0, i1, device=dev)
                a, c = short[:, i], long_[:, d - i]
                s = mat[c[:, None, :], a[None, :, :]] if swap else mat[a[:, None, :], c[None, :, :]]
                if affine:
                    m = (best2[..., i0:i1] + s).clamp_min(0.0)
                    x = torch.maximum(x1[..., i0:i1] + ext, m1[..., i0:i1] + gap + ext)
                    y = torch.maximum(y1[..., i0 + 1:i1 + 1] + ext, m1[..., i0 + 1:i1 + 1] + gap + ext)
                    h = torch.maximum(m, torch.maximum(x, y))
                else:
                    h = torch.maximum(best2[..., i0:i1] + s,
                                      torch.maximum(best1[..., i0:i1], best1[..., i0 + 1:i1 + 1]) + gap).clamp_min(0.0)
                top = torch.maximum(top, h.amax(-1))
                n = torch.zeros_like(z)
                n[..., i0 + 1:i1 + 1] = h
                best2, best1 = best1, n
                if affine:
                    m1 = torch.zeros_like(z)
                    m1[..., i0 + 1:i1 + 1] = m
                    x1, y1 = torch.full_like(z, neg), torch.full_like(z, neg)
                    x1[..., i0 + 1:i1 + 1] = x
                    y1[..., i0 + 1:i1 + 1] = y
            out[q0:q0 + 512, t0:t0 + step] = top.cpu().numpy()
    return out


def exact(case, seed):
    if case["out"] not in ("maxima", "both") or _sizes(case)[3] > 1e10:
        return None
    if case["kind"] == "database":
        targets = _database(case)
        queries = _database_queries(case, np.random.default_rng([int(seed), 1]), targets)
    else:
        queries, targets, _ = _records(case, seed)
    out = {"maxima": _maxima64(case, queries, targets)}
    if case["out"] == "both":
        out.update(hits=None, strings=None)
    return out
