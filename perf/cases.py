"""Workloads for measuring the library through its public entry points.

Each case is one call that a program using the framework makes: a scoring
call of the plug-in interface, a batch of banded regions, a protein, translated
or nucleotide search of a query batch against a resident database, seed
masking, six-frame translation, and the learned triage's inference and
gradient passes.  Sizes are those of the repository's own benchmark, tests and
presets, from one query up to the largest batch it quotes.

Inputs are synthetic and made from the seed alone: log-normal protein lengths
(median 250), Robinson background residues, planted homologs with
substitutions and indels, uniform DNA.  They are generated on the GPU and
handed over as the host arrays (or device tensors) that the entry points take.
"""
import math

import numpy as np
import torch

from saber_gb300 import synth
from saber_gb300.gpu import CudaBackend, Device
from saber_gb300.masking import Tantan
from saber_gb300.scoring import matrix as score_matrix
from saber_gb300.search import Searcher, SearchParams
from saber_gb300.translation import codon_table
from saber_gb300.triage import init_model

GPU = "cuda"


# ---- the cases ---------------------------------------------------------------
def listed():
    return [
        # one query's candidate windows through the scoring plug-in interface: the smallest call
        {"name": "windows_40", "kind": "windows", "qlen": 310, "windows": 40},
        # one small search's candidate regions from host buffers (ragged bands, few queries)
        {"name": "band_host_3k", "kind": "band", "jobs": 3001, "queries": 23, "subjects": 5003, "half_min": 4,
         "half_max": 64, "entry": "host", "bias": True},
        # the scoring stage at the size of the repository's benchmark, jobs already on the device
        {"name": "band_dev_1m", "kind": "band", "jobs": 1000000, "queries": 2000, "subjects": 200000, "half_min": 8,
         "half_max": 128, "entry": "dev", "bias": True},
        # an interactive search: one query against a mid-sized database
        {"name": "search_1x30m", "kind": "search", "queries": 1, "residues": 30000000, "preset": "default",
         "translated": False},
        # a small batch against a small database (the 64 x 20,000 blastp configuration)
        {"name": "search_64x6m", "kind": "search", "queries": 64, "residues": 6000000, "preset": "default",
         "translated": False},
        # the batched search at the benchmark's full size: the largest call
        {"name": "search_11kx150m", "kind": "search", "queries": 11000, "residues": 150000000, "preset": "default",
         "translated": False},
        # a nucleotide search (no window filter: every seed hit is extended)
        {"name": "blastn_400x150m", "kind": "blastn", "queries": 400, "bases": 150000000},
        # DNA turned into its six frames: a nucleotide database being made searchable
        {"name": "translate_30m", "kind": "translate", "bases": 30000000, "median": 900},
        # seed masking of a query batch, with the posteriors
        {"name": "tantan_600k_probs", "kind": "tantan", "residues": 600000, "probs": True},
        # seed masking at database size
        {"name": "tantan_30m", "kind": "tantan", "residues": 30000000, "probs": False},
        # the triage network over a large batch's candidate regions
        {"name": "predict_1m", "kind": "predict", "rows": 1000003},
        # one training batch's forward and backward pass (the default batch of the trainer)
        {"name": "grads_2048", "kind": "grads", "rows": 2048, "pos_weight": 78.0},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["windows", "band", "band", "search", "search", "blastn", "translate", "tantan", "predict",
                       "grads"])
    if kind == "windows":
        return {"kind": kind, "qlen": _log_int(rng, 30, 1500), "windows": _log_int(rng, 1, 400)}
    if kind == "band":
        half_max = rng.choice([24, 64, 128, 200])
        return {"kind": kind, "jobs": _log_int(rng, 500, 500000), "queries": _log_int(rng, 1, 2000),
                "subjects": _log_int(rng, 300, 100000), "half_min": rng.choice([1, 4, 8]), "half_max": half_max,
                "entry": rng.choice(["host", "dev"]), "bias": rng.choice([True, False])}
    if kind == "search":
        return {"kind": kind, "queries": _log_int(rng, 1, 1500), "residues": _log_int(rng, 2000000, 60000000),
                "preset": rng.choice(["very-fast", "fast", "default", "sensitive"]),
                "translated": rng.random() < 0.25}
    if kind == "blastn":
        return {"kind": kind, "queries": _log_int(rng, 1, 300), "bases": _log_int(rng, 5000000, 120000000)}
    if kind == "translate":
        return {"kind": kind, "bases": _log_int(rng, 100000, 20000000), "median": _log_int(rng, 300, 100000)}
    if kind == "tantan":
        return {"kind": kind, "residues": _log_int(rng, 20000, 15000000), "probs": rng.random() < 0.5}
    if kind == "predict":
        return {"kind": kind, "rows": _log_int(rng, 1000, 800000)}
    return {"kind": kind, "rows": _log_int(rng, 200, 16000), "pos_weight": float(rng.choice([1, 9, 78]))}


# ---- synthetic inputs ----------------------------------------------------------
def _gen(seed):
    g = torch.Generator(device=GPU)
    g.manual_seed(int(seed))
    return g


def _table(p, size=65536):
    """size-entry lookup table of codes with frequencies p."""
    edges = np.rint(np.cumsum(p) / np.sum(p) * size).astype(np.int64)
    return np.searchsorted(edges, np.arange(size), side="right").astype(np.uint8)


_TABLES = {}


def _tables():
    """(background residues, residues conditional on the replaced one) as GPU lookup tables."""
    if not _TABLES:
        s = score_matrix("BLOSUM62")[:20, :20].astype(np.float64)
        t = synth.BACKGROUND[:, None] * synth.BACKGROUND[None, :] * np.exp(synth.LAMBDA_U * s)
        _TABLES["bg"] = torch.from_numpy(_table(synth.BACKGROUND)).to(GPU)
        _TABLES["cond"] = torch.from_numpy(np.stack([_table(r) for r in t])).to(GPU)
    return _TABLES["bg"], _TABLES["cond"]


def _draw_codes(g, n, protein):
    if not protein:
        return torch.randint(0, 4, (n,), generator=g, device=GPU, dtype=torch.uint8)
    return _tables()[0][torch.randint(0, 65536, (n,), generator=g, device=GPU, dtype=torch.int32)]


def _protein_lengths(rng, n, hi=1500):
    return np.clip(np.rint(rng.lognormal(math.log(250.0), 0.6, size=n)), 30, hi).astype(np.int64)


def _lengths_for(total, mean, make):
    """Sequence lengths of a case: its sizes, the same for every seed."""
    return make(np.random.default_rng(17), max(1, int(total / mean)))


def _offsets(lens):
    off = np.zeros(lens.size + 1, np.uint64)
    off[1:] = np.cumsum(lens)
    return off


def _homologs(g, rng, q, qoff, which, identity, indel, protein):
    """Mutated copies of the queries `which`: (codes on the GPU, lengths)."""
    lens = torch.from_numpy((qoff[1:] - qoff[:-1]).astype(np.int64)[which]).to(GPU)
    start = torch.cumsum(lens, 0) - lens
    total = int(lens.sum())
    owner = torch.repeat_interleave(torch.arange(which.size, device=GPU), lens, output_size=total)
    first = torch.from_numpy(qoff[:-1].astype(np.int64)[which]).to(GPU)
    src = q[first[owner] + torch.arange(total, device=GPU) - start[owner]]
    keep = torch.from_numpy(identity.astype(np.float32)).to(GPU)
    sub = torch.rand(total, generator=g, device=GPU) > keep[owner]
    if protein:
        r = torch.randint(0, 65536, (total,), generator=g, device=GPU, dtype=torch.int32)
        new = _tables()[1][src.clamp(max=19).long(), r.long()]
    else:
        new = (src + torch.randint(1, 4, (total,), generator=g, device=GPU, dtype=torch.uint8)) % 4
    src = torch.where(sub, new, src)
    # an indel event inserts 1..5 residues or deletes a run of 1..5
    ev = torch.rand(total, generator=g, device=GPU) < indel
    ln = torch.randint(1, 6, (total,), generator=g, device=GPU, dtype=torch.int64)
    ins = torch.rand(total, generator=g, device=GPU) < 0.5
    gone = torch.zeros(total, dtype=torch.bool, device=GPU)
    for k in range(5):
        hit = ev & ~ins & (ln > k)
        gone[k:] |= hit[:total - k]
    count = torch.where(gone, 0, torch.where(ev & ins, 1 + ln, 1))
    at = torch.cumsum(count, 0)
    made = int(at[-1]) if total else 0
    out = torch.repeat_interleave(src, count, output_size=made)
    extra = torch.ones(made, dtype=torch.bool, device=GPU)
    extra[(at - count)[count > 0]] = False
    out = torch.where(extra, _draw_codes(g, made, protein), out)
    new_lens = torch.zeros(which.size, dtype=torch.int64, device=GPU).index_add_(0, owner, count)
    return out, new_lens.cpu().numpy()


def _related_db(g, rng, q, qoff, lens, frac, identity, indel, protein):
    """Subjects of the given lengths, a fraction of them replaced by homologs of
    random queries, in random order: (host codes, offsets, planted query or -1)."""
    n = lens.size
    n_pl = int(round(frac * n))
    which = rng.integers(0, qoff.size - 1, size=n_pl)
    ident = rng.uniform(identity[0], identity[1], size=n_pl)
    bg_lens = lens[:n - n_pl]
    bg = _draw_codes(g, int(bg_lens.sum()), protein)
    if n_pl:
        hom, hom_lens = _homologs(g, rng, q, qoff, which, ident, indel, protein)
        pool, pool_lens = torch.cat([bg, hom]), np.concatenate([bg_lens, hom_lens])
    else:
        pool, pool_lens = bg, bg_lens
    perm = rng.permutation(n)
    start = (np.cumsum(pool_lens) - pool_lens)[perm]
    out_lens = pool_lens[perm]
    off = _offsets(out_lens)
    d_len = torch.from_numpy(out_lens).to(GPU)
    total = int(out_lens.sum())
    shift = torch.from_numpy(start - off[:-1].astype(np.int64)).to(GPU)
    idx = torch.repeat_interleave(shift, d_len, output_size=total) + torch.arange(total, device=GPU)
    planted = np.concatenate([np.full(n - n_pl, -1, np.int64), which])[perm]
    return pool[idx].cpu().numpy(), off, planted


def _repeats(rng, codes, share):
    """Low-complexity stretches (period 1..6) over a share of the residues, as real sequences have."""
    n = codes.size
    m = int(n * share / 40)
    at = rng.integers(0, max(1, n - 60), size=m)
    per = rng.integers(1, 7, size=m)
    ln = rng.integers(20, 60, size=m)
    t = np.arange(60)
    idx = at[:, None] + t
    src = at[:, None] + t % per[:, None]
    ok = (t < ln[:, None]) & (idx < n) & (src < n)
    codes[idx[ok]] = codes[src[ok]]
    return codes


def _dna_of(rng, prot, lens):
    """Random-codon DNA of proteins (host codes), one record per protein."""
    ct = codon_table("standard").astype(np.int64)
    tab = np.zeros((24, 64), np.int64)
    for aa in range(24):
        c = np.flatnonzero(ct == aa)
        c = c if c.size else np.array([0])
        tab[aa] = c[np.arange(64) % c.size]
    cod = tab[np.minimum(prot, 23), rng.integers(0, 64, size=prot.size)]
    return np.stack([cod // 16, (cod // 4) % 4, cod % 4], axis=1).astype(np.uint8).reshape(-1), _offsets(3 * lens)


def _host_view(device_tensor):
    return device_tensor.cpu().numpy()


# ---- prepare / run ---------------------------------------------------------------
def prepare(case, seed):
    st = _PREPARE[case["kind"]](case, int(seed))
    st["kind"] = case["kind"]
    torch.cuda.empty_cache()
    return st


def run(state):
    return _RUN[state["kind"]](state)


def _prep_windows(case, seed):
    rng, g = np.random.default_rng(seed), _gen(seed)
    m = case["qlen"]
    q = _host_view(_draw_codes(g, m, True))
    lens = rng.integers(max(20, m // 2), 2 * m + 40, size=case["windows"])
    codes = _host_view(_draw_codes(g, int(lens.sum()), True))
    off = np.concatenate([[0], np.cumsum(lens)])
    wins = []
    for i in range(lens.size):
        w = codes[off[i]:off[i + 1]].copy()
        if i % 3 == 0:  # a related window: part of the query in place
            a = int(rng.integers(0, max(1, m // 2)))
            b = min(m, a + w.size)
            w[:b - a] = q[a:b]
        wins.append(w)
    bias = rng.integers(-1, 2, size=m).astype(np.int8)
    return {"backend": CudaBackend(0), "q": q, "bias": bias, "wins": wins, "matrix": score_matrix("BLOSUM62")}


def _run_windows(s):
    return s["backend"].score_windows(s["q"], s["bias"], s["wins"], s["matrix"], (11, 1))


def _prep_band(case, seed):
    rng, g = np.random.default_rng(seed), _gen(seed)
    qoff = _offsets(_protein_lengths(rng, case["queries"]))
    q = _draw_codes(g, int(qoff[-1]), True)
    codes, off, planted = _related_db(g, rng, q, qoff, _protein_lengths(rng, case["subjects"]), 0.10, (0.3, 0.6), 0.02,
                                      True)
    qs, ss = synth.ProteinSet(_host_view(q), qoff), synth.ProteinSet(codes, off)
    jobs = synth.band_jobs(seed + 1, qs, ss, planted, case["jobs"], half_min=case["half_min"],
                           half_max=case["half_max"])
    bias = synth.query_bias(seed + 2, qs) if case["bias"] else None
    dev = Device(0)
    dev.set_scheme(score_matrix("BLOSUM62"), 11, 1)
    dev.load_db(ss.codes, ss.offsets)
    dev.load_queries(qs.codes, qs.offsets, bias)
    st = {"dev": dev, "jobs": jobs, "entry": case["entry"]}
    if case["entry"] == "dev":
        st["d_jobs"] = torch.from_numpy(jobs.view(np.uint8).reshape(-1)).to(GPU)
        st["d_scores"] = torch.zeros(jobs.size, dtype=torch.int32, device=GPU)
    return st


def _run_band(s):
    if s["entry"] == "dev":
        s["dev"].score_band_jobs_dev(s["d_jobs"].data_ptr(), s["jobs"].size, s["d_scores"].data_ptr())
        return s["d_scores"]
    return s["dev"].score_band_jobs(s["jobs"])[0]


def _prep_search(case, seed):
    rng, g = np.random.default_rng(seed), _gen(seed)
    qlens = _protein_lengths(rng, case["queries"])
    if case["queries"] < 8:  # a short list has ordinary queries
        qlens = rng.integers(200, 500, size=case["queries"])
    qoff = _offsets(qlens)
    q = _draw_codes(g, int(qoff[-1]), True)
    lens = _lengths_for(case["residues"], 299.0, _protein_lengths)
    # a quarter of the subjects are homologs in large batches; a few dozen per query otherwise
    frac = min(0.25, 40.0 * case["queries"] / lens.size)
    codes, off, _ = _related_db(g, rng, q, qoff, lens, frac, (0.3, 0.6), 0.02, True)
    dev = Device(0)
    se = Searcher(dev, codes, off, SearchParams(case["preset"]))
    st = {"dev": dev, "se": se, "translated": case["translated"], "runs": 48}
    qh = _repeats(rng, _host_view(q), 0.02)
    if case["translated"]:
        st["q"], st["qoff"] = _dna_of(rng, qh, qlens)
        st["codon"] = codon_table("standard")
    else:
        st["q"], st["qoff"] = qh, qoff
    return st


def _hits(hits, ops, rows, runs):
    """The hit table as one array per column, in tables of a fixed size (zeros after the last hit)."""
    out = {}
    for k in hits.dtype.names:
        if k != "pad_":
            out[k] = np.zeros(rows, hits.dtype[k].str.replace("u", "i"))
            out[k][:hits.size] = hits[k]
    out["ops"] = np.zeros(rows * runs, np.int32)
    out["ops"][:ops.size] = ops.view(np.int32)
    return out


def _run_search(s):
    se, dev = s["se"], s["dev"]
    q, qoff = s["q"], s["qoff"]
    if s["translated"]:
        q, qoff = dev.translate6(q, qoff, s["codon"])
    mask, _ = se.query_mask(q, qoff)
    hits, ops, _ = dev.search(se.cparams(), se.db_codes, se.db_offsets, q, qoff, mask)
    return _hits(hits, ops, (qoff.size - 1) * se.p.max_target_seqs * se.p.max_hsps, s["runs"])


def _prep_blastn(case, seed):
    rng, g = np.random.default_rng(seed), _gen(seed)
    qoff = _offsets(rng.integers(1000, 10001, size=case["queries"]))
    q = _draw_codes(g, int(qoff[-1]), False)
    lens = _lengths_for(case["bases"], 5500.0, lambda r, n: r.integers(1000, 10001, size=n))
    frac = min(0.10, 20.0 * case["queries"] / lens.size)
    codes, off, _ = _related_db(g, rng, q, qoff, lens, frac, (0.80, 0.95), 0.01, False)
    dev = Device(0)
    se = Searcher(dev, codes, off, SearchParams.nucleotide(), nucleotide=(2, -3), gap_open=7, gap_extend=2)
    return {"dev": dev, "se": se, "translated": False, "q": _host_view(q), "qoff": qoff, "runs": 256}


def _prep_translate(case, seed):
    rng, g = np.random.default_rng(seed), _gen(seed)
    med = case["median"]
    lens = _lengths_for(case["bases"], 1.2 * med,
                        lambda r, n: np.clip(np.rint(r.lognormal(math.log(med), 0.6, size=n)), 1, 4 * med))
    lens = lens.astype(np.int64)
    nt = _host_view(_draw_codes(g, int(lens.sum()), False))
    nt[rng.integers(0, nt.size, size=nt.size // 500)] = 4  # N
    return {"dev": Device(0), "nt": nt, "off": _offsets(lens), "codon": codon_table("standard")}


def _run_translate(s):
    return s["dev"].translate6(s["nt"], s["off"], s["codon"])


def _tantan_input(case, seed):
    rng, g = np.random.default_rng(seed), _gen(seed)
    lens = _lengths_for(case["residues"], 299.0, _protein_lengths)
    codes = _repeats(rng, _host_view(_draw_codes(g, int(lens.sum()), True)), 0.05)
    return codes, _offsets(lens)


def _prep_tantan(case, seed):
    codes, off = _tantan_input(case, seed)
    return {"tantan": Tantan.protein(Device(0)), "codes": codes, "off": off, "probs": case["probs"]}


def _run_tantan(s):
    if s["probs"]:
        return s["tantan"].repeat_probs(s["codes"], s["off"])
    return s["tantan"].mask(s["codes"], s["off"])


def _triage_input(case, seed):
    """Feature rows (24 columns at the scales of real features, 8 unused), a model, labels."""
    g = _gen(seed)
    n = case["rows"]
    x = torch.randn(n, 32, generator=g, device=GPU)
    scale = torch.linspace(0.2, 4.0, 32, device=GPU)
    x = x * scale + torch.linspace(-1.0, 6.0, 32, device=GPU)
    x[:, 24:] = 0
    score = 1.5 * x[:, 0] - 0.8 * x[:, 3] + 0.5 * x[:, 7] * x[:, 9] / 8 + torch.randn(n, generator=g, device=GPU)
    y = score > torch.quantile(score[:100000], 0.95)
    rows = _host_view(x)
    return rows, _host_view(y).astype(np.uint8), init_model(seed, rows[:100000])


def _prep_triage(case, seed):
    rows, y, model = _triage_input(case, seed)
    return {"dev": Device(0), "rows": rows, "y": y, "model": model, "w": case.get("pos_weight", 1.0)}


def _run_predict(s):
    return s["dev"].triage_predict(s["model"], s["rows"])


def _run_grads(s):
    g, loss = s["dev"].triage_grads(s["model"], s["rows"], s["y"], s["w"])
    return {"grads": g, "loss": np.float64(loss)}


_PREPARE = {"windows": _prep_windows, "band": _prep_band, "search": _prep_search, "blastn": _prep_blastn,
            "translate": _prep_translate, "tantan": _prep_tantan, "predict": _prep_triage, "grads": _prep_triage}
_RUN = {"windows": _run_windows, "band": _run_band, "search": _run_search, "blastn": _run_search,
        "translate": _run_translate, "tantan": _run_tantan, "predict": _run_predict, "grads": _run_grads}


# ---- the work a pass cannot do without ---------------------------------------------
def work(case):
    k = case["kind"]
    if k == "windows":
        n = case["windows"]
        res = n * (1.25 * case["qlen"] + 20)
        return {"bytes": res + 2 * case["qlen"] + 4 * n, "flops": 11.0 * res * case["qlen"]}
    if k == "band":
        # about 60 % of a query's rows meet the window, a full band wide
        width = case["half_min"] + case["half_max"] + 1
        cells = case["jobs"] * 0.6 * 250 * width
        return {"bytes": 36.0 * case["jobs"] + 299.0 * (case["queries"] + case["subjects"]), "flops": 11 * cells}
    if k in ("search", "blastn"):
        # seed hits by the chance of a match per shape; a hit needs a 32-letter window compare
        # (protein) or an extension of about 26 positions (nucleotide)
        if k == "search":
            qn = case["queries"] * 299.0 * (2.0 if case["translated"] else 1.0)
            shapes, codes = {"very-fast": 4, "fast": 8, "default": 16, "sensitive": 8}[case["preset"]], 1.15e6
            hits = qn * case["residues"] * shapes / (codes / 8 if case["preset"] == "sensitive" else codes)
            ops = hits * 32 + 0.06 * hits * 60 * 4
            ops += 11 * min(0.0023 * hits, case["queries"] * 5000.0) * 10000
            db = case["residues"]
        else:
            qn, db = case["queries"] * 5500.0, case["bases"]
            ops = qn * db / 4.0 ** 11 * 26 * 4
        return {"bytes": db + 2 * qn, "flops": ops}
    if k == "translate":
        return {"bytes": 3.0 * case["bases"], "flops": 2.0 * case["bases"]}
    if k == "tantan":
        # forward and backward: 50 states, about five multiplications or additions each
        n = case["residues"]
        return {"bytes": n * (5.0 if case["probs"] else 2.0), "flops": n * 2.0 * 50 * 5}
    macs = 24 * 256 + 256 * 256 + 256
    n = case["rows"]
    if k == "predict":
        return {"bytes": n * (4.0 * 32 + 4) + 4 * 74561.0, "flops": 2.0 * macs * n}
    return {"bytes": n * (4.0 * 32 + 1) + 8 * 74561.0, "flops": 6.0 * macs * n}


# ---- the same outputs in 64 bits ------------------------------------------------------
def exact(case, seed):
    if case["kind"] == "tantan" and case["probs"] and case["residues"] <= 2000000:
        codes, off = _tantan_input(case, int(seed))
        return _tantan_exact(codes, off)
    if case["kind"] == "predict":
        rows, _, model = _triage_input(case, int(seed))
        p = _unpack(model)
        return torch.cat([_forward(p, torch.from_numpy(rows[i:i + 100000]).to(GPU).double())[0]
                          for i in range(0, rows.shape[0], 100000)]).cpu().numpy()
    if case["kind"] == "grads":
        rows, y, model = _triage_input(case, int(seed))
        return _grads_exact(_unpack(model), torch.from_numpy(rows).to(GPU).double(),
                            torch.from_numpy(y).to(GPU).double(), case["pos_weight"])
    return None


def _implied_lambda(s):
    """The lambda at which the entries of exp(lambda S)^-1 (20 standard residues) sum to 1."""
    def f(x):
        return np.linalg.inv(np.exp(x * s)).sum() - 1.0
    lo, hi = 0.2, 0.5
    for _ in range(200):
        mid = 0.5 * (lo + hi)
        if (f(mid) > 0) == (f(lo) > 0):
            lo = mid
        else:
            hi = mid
    return 0.5 * (lo + hi)


def _tantan_exact(codes, off, start=0.005, end=0.05, w=50, decay=0.9):
    """Posterior repeat probabilities by the forward-backward pass in 64 bits, all sequences side by side."""
    s = score_matrix("BLOSUM62").astype(np.float64)
    lr = torch.from_numpy(np.exp(_implied_lambda(s[:20, :20]) * s)).to(GPU)
    lr = torch.cat([lr, torch.zeros(24, 1, dtype=torch.float64, device=GPU)], 1)  # column 24: no partner
    b2f = torch.from_numpy(start * (1 - decay) / (1 - decay ** w) * decay ** np.arange(w)).to(GPU)
    lens = (off[1:] - off[:-1]).astype(np.int64)
    order = np.argsort(-lens, kind="stable")
    lens = lens[order]
    nseq, longest = lens.size, int(lens[0])
    first = torch.from_numpy(off[:-1].astype(np.int64)[order]).to(GPU)
    x = torch.from_numpy(np.concatenate([codes, np.zeros(longest, np.uint8)])).to(GPU)
    live = [int(np.searchsorted(-lens, -p, side="left")) for p in range(longest)]  # sequences longer than p

    def emit(p, n):
        at = first[:n, None] + p - 1 - torch.arange(w, device=GPU)
        part = torch.where(torch.arange(w, device=GPU) < p, x[at.clamp(min=0)].long(), 24)
        return lr[x[first[:n] + p].long()[:, None], part]

    b = torch.ones(nseq, dtype=torch.float64, device=GPU)
    f = torch.zeros(nseq, w, dtype=torch.float64, device=GPU)
    rows, scales = [], []
    for p in range(longest):
        n = live[p]
        nf = (b[:n, None] * b2f + f[:n] * (1 - end)) * emit(p, n)
        nb = b[:n] * (1 - start) + f[:n].sum(1) * end
        sc = 1.0 / (nb + nf.sum(1))
        b, f = nb * sc, nf * sc[:, None]
        rows.append((b, f))
        scales.append(sc)
    out = torch.zeros(codes.size, dtype=torch.float64, device=GPU)
    b = torch.ones(nseq, dtype=torch.float64, device=GPU)
    f = torch.full((nseq, w), end, dtype=torch.float64, device=GPU)
    for p in range(longest - 1, -1, -1):
        n = live[p]
        fb, ff = rows[p]
        pf = (ff * f[:n]).sum(1)
        out[first[:n] + p] = pf / (fb * b[:n] + pf)
        if p:
            be = emit(p, n) * f[:n]
            sc = scales[p]
            nb = ((1 - start) * b[:n] + (b2f * be).sum(1)) * sc
            f[:n] = ((1 - end) * be + end * b[:n, None]) * sc[:, None]
            b[:n] = nb
    return out.cpu().numpy()


def _unpack(model):
    """Model layout: W1[32][256], b1, W2[256][256], b2, W3, b3, mu[32], isd[32]; weights as bf16."""
    m = torch.from_numpy(model).to(GPU)
    cut = np.cumsum([32 * 256, 256, 256 * 256, 256, 256, 1, 32, 32])
    w1, b1, w2, b2, w3, b3, mu, isd = (m[a:b] for a, b in zip(np.concatenate([[0], cut[:-1]]), cut))
    bf = lambda t: t.bfloat16().double()  # noqa: E731
    return dict(w1=bf(w1).reshape(32, 256), b1=b1.double(), w2=bf(w2).reshape(256, 256), b2=b2.double(), w3=bf(w3),
                b3=b3.double(), mu=mu.double(), isd=isd.double())


def _forward(p, x):
    xn = (x - p["mu"]) * p["isd"]
    xn[:, 24:] = 0
    h1 = torch.relu(xn @ p["w1"] + p["b1"])
    h2 = torch.relu(h1 @ p["w2"] + p["b2"])
    return h2 @ p["w3"] + p["b3"], xn, h1, h2


def _grads_exact(p, x, y, pos_weight):
    z, xn, h1, h2 = _forward(p, x)
    n = x.shape[0]
    wt = torch.where(y > 0, pos_weight, 1.0).double()
    loss = (wt * (torch.log1p(torch.exp(-z.abs())) + z.clamp(min=0) - y * z)).sum() / n
    dz = wt * (torch.sigmoid(z) - y) / n
    dh2 = dz[:, None] * p["w3"] * (h2 > 0)
    dh1 = (dh2 @ p["w2"].T) * (h1 > 0)
    zero = torch.zeros(64, dtype=torch.float64, device=GPU)
    g = torch.cat([(xn.T @ dh1).reshape(-1), dh1.sum(0), (h1.T @ dh2).reshape(-1), dh2.sum(0), h2.T @ dz,
                   dz.sum().reshape(1), zero])
    return {"grads": g.cpu().numpy(), "loss": np.float64(loss.item())}
