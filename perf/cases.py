"""Performance cases of the library: what its users call, over the sizes they call it with.

Every case goes through one public entry point of g3sa_b200 (`call`):

  extend   Context.extend_batch / capture_batch  batches of ksw_extend2 jobs in device memory
  seeds    Context.extend_seeds                  left + right extension of seeds with band retry
  stream   Context.extend_seeds_stream           the same from host memory, chunk by chunk
  chains   Context.chain2aln                     the chain level, whole reads
  global   Context.global_batch                  banded global alignment with CIGAR, NM and MD
  align    Context.align2_batch                  striped local alignment of seed windows
  filter   Context.flt_chained_seeds             the seed filter of long reads

All results are whole numbers that the reference's algorithm fixes, so they are compared bit for
bit.  Inputs are seeded synthetic ones in the shapes of the benchmark's workloads and the tests.
"""
import math

import numpy as np
import torch

import g3sa_b200 as g
from g3sa_b200 import chains as gc
from g3sa_b200 import learn

# Scorings in use: BWA's defaults, unequal gap costs, and a doubled match score (the tests' three).
SCORES = {
    "bwa": {"a": 1},
    "uneven": {"a": 1, "o_del": 5, "e_del": 2, "o_ins": 7, "e_ins": 1},
    "match2": {"a": 2, "b": 3, "o_del": 5, "e_del": 2, "o_ins": 4, "e_ins": 3},
}
# Width classes as a program keeps them from one Context.autotune of its workload: 100-250 base
# reads in the length order, and long segments at bands up to 100 and up to 500.
TILES = {
    "reads": [(32, 1, 2, 0, 32), (56, 1, 2, 0, 32), (88, 1, 2, 0, 32), (128, 1, 2, 0, 32), (168, 1, 2, 0, 32),
              (200, 1, 2, 0, 32), (232, 1, 2, 0, 8), (2147483647, 32, 9, 0, 1)],
    "long100": [(w, 32, 256, 0, 1) for w in (696, 1208, 1896, 2760, 3624, 4312, 5000)] + [(2147483647, 32, 9, 0, 1)],
    "long500": [(w, 32, 1024, 0, 1) for w in (696, 1208, 1896, 2760, 3624, 4312, 5000)] + [(2147483647, 32, 9, 0, 1)],
}
OPS = 8     # integer operations of a DP cell (M: add and select; H: max3; row max; E and F: two each)


def listed():
    return [
        # the extensions of a few reads, as an interactive tool or a tail of a run sends them
        {"name": "extend-few", "call": "extend", "kind": 2, "units": 32, "w": 100, "unrelated": 0.2, "score": "bwa",
         "int16": True, "schedule": "sorted", "tiles": "", "graph": False},
        # an ordinary batch with other gap costs than BWA's and a narrower band, default classes
        {"name": "extend-batch", "call": "extend", "kind": 2, "units": 10007, "w": 50, "unrelated": 0.2,
         "score": "uneven", "int16": True, "schedule": "sorted", "tiles": "", "graph": False},
        # the benchmark's batch: about a million uneven jobs, tuned classes, learned order, one graph
        {"name": "extend-million", "call": "extend", "kind": 2, "units": 500000, "w": 100, "unrelated": 0.2,
         "score": "bwa", "int16": True, "schedule": "learned", "tiles": "reads", "graph": True},
        # long segments in int32, tuned classes
        {"name": "long-w100", "call": "extend", "kind": 4, "units": 20000, "w": 100, "unrelated": 0.0, "score": "bwa",
         "int16": False, "schedule": "sorted", "tiles": "long100", "graph": False},
        # long segments with a wide band on a context as it is created
        {"name": "long-w500-default", "call": "extend", "kind": 4, "units": 1500, "w": 500, "unrelated": 0.0,
         "score": "bwa", "int16": True, "schedule": "sorted", "tiles": "", "graph": False},
        # the seeds of a small batch of reads, with band retry
        {"name": "seeds-2k", "call": "seeds", "units": 2003, "w": 100, "unrelated": 0.2, "score": "bwa"},
        # a run's seeds from pinned host memory in 64k chunks, the last one ragged
        {"name": "stream-500k", "call": "stream", "units": 500000, "w": 100, "unrelated": 0.2, "score": "bwa",
         "chunk": 65536, "schedule": "learned"},
        # the chain level of a batch of reads
        {"name": "chains-8k", "call": "chains", "reads": 8000, "w": 100, "score": "bwa"},
        # the traceback stage's alignments: CIGAR, NM and MD
        {"name": "global-200k", "call": "global", "n": 200000, "max_len": 250, "md": True, "score": "bwa"},
        # a few hundred pairs, CIGAR only
        {"name": "global-few", "call": "global", "n": 311, "max_len": 250, "md": False, "score": "bwa"},
        # seed windows of a large batch with their start positions
        {"name": "align-200k", "call": "align", "n": 200000, "xtra": g.KSW_XSTART, "score": "bwa"},
        # the seed filter of a batch of long reads
        {"name": "filter-1k", "call": "filter", "reads": 1200, "w": 100, "score": "bwa"},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    call = rng.choice(["extend", "extend", "long", "seeds", "stream", "chains", "global", "align", "filter"])
    score = rng.choice(["bwa", "bwa", "uneven", "match2"])
    if call == "extend":
        schedule = rng.choice(["sorted", "learned"])
        return {"call": "extend", "kind": rng.choice([1, 2, 2]), "units": _log_int(rng, 16, 400000),
                "w": rng.randint(10, 100), "unrelated": round(rng.uniform(0.0, 0.5), 2), "score": score,
                "int16": True, "schedule": schedule, "tiles": rng.choice(["", "reads"]), "graph": schedule == "learned"}
    if call == "long":
        w = rng.choice([rng.randint(10, 100), rng.randint(101, 500)])
        return {"call": "extend", "kind": 4, "units": _log_int(rng, 20, 1500 if w > 100 else 6000), "w": w,
                "unrelated": 0.0, "score": score, "int16": rng.choice([True, False]), "schedule": "sorted",
                "tiles": rng.choice(["", "long100" if w <= 100 else "long500"]), "graph": False}
    if call == "seeds":
        return {"call": "seeds", "units": _log_int(rng, 16, 200000), "w": rng.randint(10, 100),
                "unrelated": round(rng.uniform(0.0, 0.5), 2), "score": score}
    if call == "stream":
        return {"call": "stream", "units": _log_int(rng, 20000, 450000), "w": rng.randint(10, 100),
                "unrelated": round(rng.uniform(0.0, 0.5), 2), "score": score, "chunk": rng.choice([32768, 65536]),
                "schedule": rng.choice(["sorted", "learned"])}
    if call == "chains":
        return {"call": "chains", "reads": _log_int(rng, 20, 8000), "w": rng.randint(20, 100), "score": score}
    if call == "global":
        return {"call": "global", "n": _log_int(rng, 100, 190000), "max_len": rng.randint(20, 250),
                "md": rng.choice([True, False]), "score": score}
    if call == "align":
        xtra = rng.choice([0, g.KSW_XSTART, g.KSW_XSTART, g.KSW_XSUBO | g.KSW_XSTART | 19])
        return {"call": "align", "n": _log_int(rng, 100, 190000), "xtra": xtra, "score": score}
    return {"call": "filter", "reads": _log_int(rng, 20, 1200), "w": rng.randint(20, 100), "score": score}


# ---- inputs ------------------------------------------------------------------------------------

def _score(case):
    return g.default_score(**SCORES[case["score"]])


def _opt(case):
    return g.default_opt(w=case["w"], **SCORES[case["score"]])


def _synth(case, kind, seed):
    kw = {k: v for k, v in SCORES[case["score"]].items() if k != "b"}
    return g.synth(kind, case["units"], seed=seed, w=case["w"], unrelated=case["unrelated"], **kw)


def _max_jobs(case):
    """Result slots of a batch: a seed gives a left and a right job unless it ends its read."""
    return case["units"] * (2 if case["kind"] == 2 else 1)


def _dev(a, records=None):
    """A record array in device memory, with room for `records` of them."""
    if records is not None:
        assert len(a) <= records
        a = np.concatenate([a, np.zeros(records - len(a), a.dtype)])
    return torch.from_numpy(np.ascontiguousarray(a).view(np.uint8).copy()).cuda()


def _pin(a):
    return torch.from_numpy(np.ascontiguousarray(a).view(np.uint8).copy()).pin_memory()


_weights = []


def _learned(ctx):
    """The cost model's weights, trained once by this program (learn.train on a small trace set)."""
    if not _weights:
        t = g.Context(0)
        learn.train(t, n_train=60000, seed_train=91, epochs=2, kind=2)
        _weights.append(t.mlp_params())
        t.close()
    ctx.mlp_set_params(_weights[0])


def _mutate(rng, seq, owner, rate, n_owner):
    """Each base of `seq` (of sequence owner[k]) substituted, deleted or followed by an insertion
    at rate[k]; returns the new concatenation and each sequence's new length."""
    u = rng.random(len(seq))
    s = seq.copy()
    sub = u < rate * 0.7
    s[sub] = rng.integers(0, 4, int(sub.sum()))
    dele = (u >= rate * 0.7) & (u < rate * 0.85)
    extra = np.where((u >= rate * 0.85) & (u < rate), rng.integers(1, 4, len(seq)), 0)
    counts = np.where(dele, 0, 1 + extra)
    out = np.repeat(s, counts)
    is_ins = np.ones(len(out), bool)
    is_ins[(np.cumsum(counts) - counts)[~dele]] = False
    out[is_ins] = rng.integers(0, 4, int(is_ins.sum()))
    return out.astype(np.uint8), np.bincount(owner, weights=counts, minlength=n_owner).astype(np.int64)


def _with_n(rng, q, qo, ql, frac):
    """A few N codes in a share of the sequences."""
    k = np.repeat(np.nonzero((rng.random(len(ql)) < frac) & (ql > 0))[0], 2)
    q[qo[k] + (rng.random(len(k)) * ql[k]).astype(np.int64)] = 4


def _pairs(q, ql, t, tl):
    """Queries and targets side by side in one code buffer, and their jobs."""
    n = len(ql)
    qo, to = np.cumsum(ql) - ql, np.cumsum(tl) - tl
    total = ql + tl
    base = np.cumsum(total) - total
    u8 = np.empty(max(int(total.sum()), 1), np.uint8)
    u8[np.repeat(base - qo, ql) + np.arange(len(q))] = q
    u8[np.repeat(base + ql - to, tl) + np.arange(len(t))] = t
    jobs = np.zeros(n, g.JOB_DT)
    jobs["q_off"], jobs["t_off"], jobs["qlen"], jobs["tlen"] = base, base + ql, ql, tl
    return u8, jobs


def _global_pairs(n, max_len, seed):
    """Region pairs: up to 250 bases, a few edits each, bands as the stage infers them."""
    rng = np.random.default_rng(seed)
    ql = rng.integers(0, max_len, n)
    q = rng.integers(0, 4, int(ql.sum())).astype(np.uint8)
    _with_n(rng, q, np.cumsum(ql) - ql, ql, 0.1)
    rate = np.minimum(rng.integers(0, 6, n) / np.maximum(ql, 1), 0.3)
    t, tl = _mutate(rng, q, np.repeat(np.arange(n), ql), np.repeat(rate, ql), n)
    u8, jobs = _pairs(q, ql, t, tl)
    jobs["w"] = rng.choice([5, 10, 20, 50], n)
    return u8, jobs


def _windows(n, seed):
    """Seed windows: a seed of 19-59 bases with up to 50 bases either side, half the flanks related."""
    rng = np.random.default_rng(seed)
    seed_len = rng.integers(19, 60, n)
    left, right = rng.integers(0, 51, n), rng.integers(0, 51, n)
    ql = left + seed_len + right
    qo = np.cumsum(ql) - ql
    q = rng.integers(0, 4, int(ql.sum())).astype(np.uint8)
    owner = np.repeat(np.arange(n), ql)
    pos = np.arange(len(q)) - np.repeat(qo, ql)
    core = (pos >= left[owner]) & (pos < (left + seed_len)[owner])
    related = rng.random(n) < 0.5
    t, tl = _mutate(rng, q, owner, np.where(core, 0.02, (rng.random(n) * 0.1)[owner]), n)
    # an unrelated flank: the same number of bases, all drawn anew (the seed's share stays)
    t_owner = np.repeat(np.arange(n), tl)
    t_pos = np.arange(len(t)) - np.repeat(np.cumsum(tl) - tl, tl)
    flank = (t_pos < left[t_owner]) | (t_pos >= (tl - right)[t_owner])
    anew = flank & ~related[t_owner]
    t[anew] = rng.integers(0, 4, int(anew.sum()))
    _with_n(rng, q, qo, ql, 0.05)
    return _pairs(q, ql, t, tl)


def prepare(case, seed):
    call = case["call"]
    ctx = g.Context(0)
    s = {"case": case, "ctx": ctx}
    if call == "extend":
        wl = _synth(case, case["kind"], seed)
        codes, nmask = wl.planes()
        if not case["int16"]:
            ctx.set_int16(False)            # every score in int32
        if case["tiles"]:
            ctx.set_tiles(TILES[case["tiles"]])
        s.update(score=_score(case), n=wl.n, jobs=_dev(wl.jobs), codes=_dev(codes), nmask=_dev(nmask),
                 out=torch.zeros((_max_jobs(case), 6), dtype=torch.int32, device="cuda"),
                 status=torch.zeros(_max_jobs(case), dtype=torch.int32, device="cuda"),
                 mq=int(wl.jobs["qlen"].max()), mt=int(wl.jobs["tlen"].max()),
                 schedule=g.SCHED_LEARNED if case["schedule"] == "learned" else g.SCHED_SORTED)
        if case["schedule"] == "learned":
            _learned(ctx)
        if case["graph"]:
            s["graph"] = ctx.capture_batch(s["score"], s["jobs"], s["n"], s["codes"], s["nmask"], s["out"],
                                           s["status"], s["mq"], s["mt"], schedule=s["schedule"])
    elif call in ("seeds", "stream"):
        wl = _synth(case, 2, seed)
        codes, nmask = wl.planes()
        ds = g.device_seeds(wl.seeds)
        n = len(ds)
        s.update(opt=_opt(case), n=n, mq=int(wl.seeds["l_query"].max()), n_bases=len(wl.u8),
                 mt=int((wl.seeds["rmax1"] - wl.seeds["rmax0"]).max()))
        words = n * g.REG_DT.itemsize // 4
        if call == "seeds":
            s.update(seeds=_dev(ds), codes=_dev(codes), nmask=_dev(nmask),
                     regs=torch.zeros(words, dtype=torch.int32, device="cuda"),
                     status=torch.zeros(n, dtype=torch.int32, device="cuda"))
        else:
            s.update(seeds=_pin(ds), codes=_pin(codes), nmask=_pin(nmask),
                     regs=torch.zeros(words, dtype=torch.int32).pin_memory(),
                     status=torch.zeros(n, dtype=torch.int32).pin_memory(),
                     schedule=g.SCHED_LEARNED if case["schedule"] == "learned" else g.SCHED_SORTED)
            if case["schedule"] == "learned":
                _learned(ctx)
    elif call in ("chains", "filter"):
        if call == "chains":
            wl = gc.synth_chains(case["reads"], seed=seed, a=SCORES[case["score"]]["a"])
        else:
            wl = gc.synth_chains(case["reads"], seed=seed, a=SCORES[case["score"]]["a"], div=0.03,
                                 read_lens=(800, 1000, 1500, 2000))
        codes, nmask = wl.planes()
        nr, ns = len(wl.reads), len(wl.seeds)
        max_chains, max_seeds = 3 * nr, (10 if call == "chains" else 48) * nr
        s.update(opt=_opt(case), l_pac=wl.l_pac, ref_off=wl.ref_off, anns=_dev(wl.anns), n_anns=len(wl.anns),
                 reads=_dev(wl.reads), n_reads=nr, chains=_dev(wl.chains, max_chains), n_chains=len(wl.chains),
                 seeds=_dev(wl.seeds, max_seeds), n_seeds=ns, codes=_dev(codes), nmask=_dev(nmask),
                 status=torch.zeros(nr, dtype=torch.int32, device="cuda"))
        if call == "chains":
            s.update(regs=torch.zeros(max_seeds * gc.ALNREG_DT.itemsize // 4, dtype=torch.int32, device="cuda"),
                     nregs=torch.zeros(nr, dtype=torch.int32, device="cuda"))
        else:
            s.update(sw=torch.zeros(max_seeds, dtype=torch.int32, device="cuda"), chains_io=torch.empty_like(s["chains"]),
                     seeds_io=torch.empty_like(s["seeds"]))
    elif call == "global":
        u8, jobs = _global_pairs(case["n"], case["max_len"], seed)
        codes, nmask = g.pack_planes(u8)
        n = len(jobs)
        s.update(score=_score(case), n=n, jobs=_dev(jobs), codes=_dev(codes), nmask=_dev(nmask),
                 mq=int(jobs["qlen"].max()), mt=int(jobs["tlen"].max()), mw=int(jobs["w"].max()), slots=64, md=128,
                 d_score=torch.zeros(n, dtype=torch.int32, device="cuda"),
                 cigar=torch.zeros((n, 64), dtype=torch.int32, device="cuda"),
                 n_cigar=torch.zeros(n, dtype=torch.int32, device="cuda"),
                 status=torch.zeros(n, dtype=torch.int32, device="cuda"),
                 d_nm=torch.zeros(n, dtype=torch.int32, device="cuda") if case["md"] else None,
                 d_md=torch.zeros((n, 128), dtype=torch.uint8, device="cuda") if case["md"] else None)
    else:
        u8, jobs = _windows(case["n"], seed)
        codes, nmask = g.pack_planes(u8)
        n = len(jobs)
        s.update(score=_score(case), n=n, jobs=_dev(jobs), codes=_dev(codes), nmask=_dev(nmask),
                 mt=int(jobs["tlen"].max()), out=torch.zeros((n, 7), dtype=torch.int32, device="cuda"),
                 status=torch.zeros(n, dtype=torch.int32, device="cuda"))
    return s


# ---- one pass ----------------------------------------------------------------------------------

def run(s):
    case, ctx = s["case"], s["ctx"]
    call = case["call"]
    if call == "extend":
        if case["graph"]:
            s["graph"].launch()
        else:
            ctx.extend_batch(s["score"], s["jobs"], s["n"], s["codes"], s["nmask"], s["out"], s["status"], s["mq"],
                             s["mt"], schedule=s["schedule"])
        return s["out"], s["status"]
    if call == "seeds":
        ctx.extend_seeds(s["opt"], s["seeds"], s["n"], s["codes"], s["nmask"], s["regs"], s["status"], s["mq"],
                         s["mt"])
        return s["regs"], s["status"]
    if call == "stream":
        ctx.extend_seeds_stream(s["opt"], s["seeds"], s["codes"], s["nmask"], s["n_bases"], s["regs"], s["status"],
                                s["mq"], s["mt"], chunk=case["chunk"], schedule=s["schedule"])
        return s["regs"], s["status"]
    if call == "chains":
        ctx.chain2aln(s["opt"], s["l_pac"], s["ref_off"], s["anns"], s["n_anns"], s["reads"], s["n_reads"],
                      s["chains"], s["n_chains"], s["seeds"], s["n_seeds"], s["codes"], s["nmask"], s["regs"],
                      s["nregs"], s["status"])
        return s["regs"], s["nregs"], s["status"]
    if call == "global":
        ctx.global_batch(s["score"], s["jobs"], s["n"], s["codes"], s["nmask"], s["mq"], s["mt"], s["mw"],
                         s["d_score"], s["cigar"], s["slots"], s["n_cigar"], s["status"], d_nm=s["d_nm"],
                         d_md=s["d_md"], md_stride=s["md"] if case["md"] else 0)
        return s["d_score"], s["cigar"], s["n_cigar"], s["status"], s["d_nm"], s["d_md"]
    if call == "align":
        ctx.align2_batch(s["score"], s["jobs"], s["n"], s["codes"], s["nmask"], case["xtra"], s["mt"], s["out"],
                         s["status"])
        return s["out"], s["status"]
    # the filter changes its chains and seeds in place: a pass starts from a fresh copy
    s["chains_io"].copy_(s["chains"])
    s["seeds_io"].copy_(s["seeds"])
    ctx.flt_chained_seeds(s["opt"], 0, s["l_pac"], s["ref_off"], s["anns"], s["n_anns"], s["reads"], s["n_reads"],
                          s["chains_io"], s["n_chains"], s["seeds_io"], s["n_seeds"], s["codes"], s["nmask"],
                          s["status"], d_sw_score=s["sw"])
    return s["chains_io"], s["seeds_io"], s["sw"], s["status"]


# ---- what a pass cannot do without -------------------------------------------------------------

def _cells_per_job(case):
    """Mean DP cells of a synthetic extension job (the oracle's counts at a few bands)."""
    w, related = case["w"], 1.0 - case["unrelated"]
    if case["kind"] == 4:
        return np.interp(w, [20, 100, 200, 500], [75.8e3, 367e3, 709e3, 1550e3])
    if case["kind"] == 1:
        return np.interp(w, [20, 100], [2900, 9550]) * (0.15 + 0.85 * related)
    return np.interp(w, [20, 50, 100], [2660, 5250, 6690]) * (0.1 + 0.9 * related)


def work(case):
    call = case["call"]
    if call in ("extend", "seeds", "stream"):
        n = case["units"]
        kind = case.get("kind", 2)
        jobs = n if kind != 2 else 1.98 * n
        bases = {1: 253, 2: 456, 4: 3925}[kind] * n
        cells = jobs * _cells_per_job({**case, "kind": kind})
        per = 24 + 28 if call == "extend" else 24 + 22
        return {"bytes": bases * 3 / 8 + jobs * per, "flops": OPS * cells}
    if call == "chains":
        return {"bytes": case["reads"] * (150 * 3 / 8 + 24 + 2 * 16 + 5 * 24 + 3 * 56), "flops": OPS * case["reads"] * 8500}
    if call == "filter":
        return {"bytes": case["reads"] * (1300 * 3 / 8 + 24 + 2 * 16 + 24 * 48),
                "flops": OPS * case["reads"] * 24 * 14000}
    n = case["n"]
    if call == "global":
        ql = case["max_len"] / 2
        cells = n * ql * min(ql, 31.0)
        return {"bytes": n * (ql * 2 * 3 / 8 + 24 + 40 + (24 if case["md"] else 0)), "flops": OPS * cells}
    passes = 1.9 if case["xtra"] & g.KSW_XSTART else 1.0
    return {"bytes": n * (180 * 3 / 8 + 24 + 32), "flops": OPS * n * 8300 * passes}


def tolerance(case):
    return "exact"


# ---- the extension in plain numpy --------------------------------------------------------------

def exact(case, seed):
    """ksw_extend2 of every job of a small batch in 64-bit numpy: all jobs' rows together, F as a
    running maximum along the row.  None for the other calls and for batches that take too long."""
    if case["call"] != "extend" or case["kind"] == 4 or case["units"] > 1500:
        return None
    wl = _synth(case, case["kind"], seed)
    sc = _score(case)[0]
    mat = np.asarray(sc["mat"], np.int64).reshape(5, 5)
    o_del, e_del, o_ins, e_ins = (int(sc[k]) for k in ("o_del", "e_del", "o_ins", "e_ins"))
    zdrop, bonus, best_match = int(sc["zdrop"]), int(sc["end_bonus"]), int(mat.max())
    jb = wl.jobs
    n = len(jb)
    ql, tl, h0 = (jb[k].astype(np.int64) for k in ("qlen", "tlen", "h0"))
    Q, T = int(ql.max()), int(tl.max())
    col = np.arange(Q + 2)

    def bases(off, length, rev, width):
        k = np.arange(width)[None, :]
        at = np.where(rev[:, None], length[:, None] - 1 - k, k)
        ok = (at >= 0) & (at < length[:, None])
        return np.where(ok, wl.u8[np.where(ok, off[:, None].astype(np.int64) + at, 0)], 4).astype(np.int64)

    q = bases(jb["q_off"], ql, (jb["flags"] & g.JOB_QREV) != 0, Q)
    t = bases(jb["t_off"], tl, (jb["flags"] & g.JOB_TREV) != 0, T)
    w = jb["w"].astype(np.int64)
    for o, e in ((o_ins, e_ins), (o_del, e_del)):
        w = np.minimum(w, np.maximum(((ql * best_match + bonus - o) / e + 1.0).astype(np.int64), 1))
    # row -1: h0, then the gap along the query
    H = np.maximum(h0[:, None] - (o_ins + e_ins * col)[None, :], 0)
    H[:, 0] = h0
    H[col[None, :] > np.maximum(ql, 1)[:, None]] = 0
    E = np.zeros_like(H)
    best, bi, bj, max_off = h0.copy(), np.full(n, -1), np.full(n, -1), np.zeros(n, np.int64)
    gscore, gi = np.full(n, -1), np.full(n, -1)
    beg, end, live = np.zeros(n, np.int64), ql.copy(), tl > 0
    rows = np.arange(n)
    for i in range(T):
        if not live.any():
            break
        b = np.maximum(beg, i - w)
        e = np.minimum(np.minimum(end, i + w + 1), ql)
        h1 = np.where(b == 0, np.maximum(h0 - (o_del + e_del * (i + 1)), 0), 0)
        inside = (col[None, :-2] >= b[:, None]) & (col[None, :-2] < e[:, None])
        Hc, Ec = H[:, :Q], E[:, :Q]
        M = np.where(Hc != 0, Hc + mat[t[:, i][:, None], q], 0)
        gap = np.where(inside, np.maximum(M - (o_ins + e_ins), 0), 0)
        run_max = np.maximum.accumulate(gap + e_ins * col[None, :Q], axis=1)
        F = np.zeros_like(M)
        F[:, 1:] = np.maximum(run_max[:, :-1] - e_ins * col[None, :Q - 1], 0)
        hv = np.maximum(np.maximum(M, Ec), F)
        new_e = np.maximum(Ec - e_del, np.maximum(M - (o_del + e_del), 0))
        hin = np.where(inside, hv, -1)
        m = np.maximum(hin.max(axis=1), 0)
        mj = Q - 1 - np.argmax(hin[:, ::-1], axis=1)
        full = e > b
        last = np.where(full, hv[rows, np.maximum(e - 1, 0)], h1)
        sel = inside & live[:, None]
        shifted = np.concatenate([np.zeros((n, 1), np.int64), hv[:, :-1]], axis=1)
        shifted[rows, np.minimum(b, Q - 1)] = h1
        H[:, :Q] = np.where(sel, shifted, Hc)
        E[:, :Q] = np.where(sel, new_e, Ec)
        put = live & full
        H[rows[put], e[put]] = last[put]
        E[rows[put], e[put]] = 0
        if (live & ~full).any():
            k = rows[live & ~full]
            H[k, np.maximum(e[k], 0)] = h1[k]
            E[k, np.maximum(e[k], 0)] = 0
        reach = live & (np.where(full, e, b) == ql)
        gi = np.where(reach & (last >= gscore), i, gi)
        gscore = np.where(reach, np.maximum(gscore, last), gscore)
        zero = live & (m == 0)
        up = live & ~zero & (m > best)
        max_off = np.where(up, np.maximum(max_off, np.abs(mj - i)), max_off)
        di, dj = i - bi, mj - bj
        drop = np.where(di > dj, best - m - (di - dj) * e_del, best - m - (dj - di) * e_ins)
        stop = live & ~zero & ~up & (zdrop > 0) & (drop > zdrop)
        best, bi, bj = np.where(up, m, best), np.where(up, i, bi), np.where(up, mj, bj)
        live = live & ~zero & ~stop
        # the next row's band: trimmed of zero entries at both ends
        filled = (H != 0) | (E != 0)
        right = col[None, :] <= e[:, None]
        ahead = filled & (col[None, :] >= b[:, None]) & (col[None, :] < e[:, None])
        nb = np.where(ahead.any(axis=1), np.argmax(ahead, axis=1), e)
        back = filled & (col[None, :] >= nb[:, None]) & right
        ne = np.where(back.any(axis=1), Q + 1 - np.argmax(back[:, ::-1], axis=1), nb - 1)
        beg, end = np.where(live, nb, beg), np.where(live, np.minimum(ne + 2, ql), end)
        live = live & (i + 1 < tl)
    out = np.zeros((_max_jobs(case), 6), np.int64)
    out[:n] = np.stack([best, bj + 1, bi + 1, gi + 1, gscore, max_off], axis=1)
    return out, np.zeros(len(out), np.int64)
