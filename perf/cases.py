"""Workloads of the MSV filter and the filter stages after it, for timing.

A case is one call that a program searching protein sequences makes through
``cudahmmsearch_gb300.api``, by ``kind``:

  dropin   p7_MSVFilter's drop-in, called for one sequence after another as an unmodified program does
  search   one profile against a resident database, results left on the GPU
  batch    many profiles against one resident database (a captured batch, replayed)
  bias     the bias filter on a list of survivors of a resident database
  vit      the ViterbiFilter on a list of survivors of a resident database
  host     one profile against a database in host memory (upload, sort, search, results)
  filters  the whole filter cascade (MSV, bias, ViterbiFilter) from host memory

Sequences: residues i.i.d. from HMMER's amino background with 0.5% X, lognormal
lengths (median 300, sigma 0.7, as protein databases have), a share of them
carrying a stretch emitted from the profile's match states. ``long_frac`` of the
lengths are uniform in [5000, 35000] (a database with titin-like proteins).
"""
import math
import os

import numpy as np
import torch

from cudahmmsearch_gb300 import api
from cudahmmsearch_gb300 import formats as F

GOLDEN = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "tests", "golden")
# Models with all parts of a profile in the repository: three of Pfam's (as
# HMMER's tutorial ships them) and sampled ones. Name: model length.
CASCADE = {"tut_fn3": 86, "tut_globins4": 149, "tut_pkinase": 260, "m50_s1": 50, "m200_s1": 200, "m400_s1": 400,
           "m777_s3": 777}
# Models with a ViterbiFilter part only.
VITERBI = dict(CASCADE, vitw5_m157_s5=157, vitw9_m285_s9=285, vitw13_m413_s13=413, vitw20_m637_s20=637,
               vitw28_m893_s28=893, vitmid_m1100_s4=1100, m1500_s2=1500, m2400_s1=2400, vitwide_m4000_s7=4000)
MEAN_LEN = 383.0                       # of the lognormal lengths
MOST_CELLS = 400 * 2_000_000 * MEAN_LEN  # the largest listed case


def listed():
    return [
        # the drop-in inside an unmodified program's loop: one call per sequence, launch and copies count
        {"name": "dropin_m200", "kind": "dropin", "M": 200, "n": 16, "lmax": 5000},
        # a domain model against a handful of bacterial proteomes
        {"name": "search_m200_20k", "kind": "search", "M": 200, "n": 20_000, "lmax": 5000, "long_frac": 0.0},
        # a short domain model (most of Pfam) against a Swiss-Prot sized database
        {"name": "search_m86_500k", "kind": "search", "M": 86, "n": 500_000, "lmax": 35000, "long_frac": 0.0},
        # one query at throughput scale: the benchmark's default workload
        {"name": "search_m400_2m", "kind": "search", "M": 400, "n": 2_000_000, "lmax": 35000, "long_frac": 0.0},
        # a multi-domain protein model
        {"name": "search_m1501_150k", "kind": "search", "M": 1501, "n": 150_000, "lmax": 35000, "long_frac": 0.0},
        # length extremes: a long model, a tenth of the targets long
        {"name": "search_m2400_20k_long", "kind": "search", "M": 2400, "n": 20_000, "lmax": 35000, "long_frac": 0.1},
        # a profile library against a small resident database (the batched path's own range)
        {"name": "batch_48x20k", "kind": "batch", "nprof": 48, "n": 20_000, "lmax": 35000},
        # the MSV survivors of a large search (2% and the homologs of 1,000,000 sequences)
        {"name": "bias_m260_40k", "kind": "bias", "model": "tut_pkinase", "n": 200_000, "nlist": 40_000},
        # the sequences past the bias filter
        {"name": "vit_m260_40k", "kind": "vit", "model": "tut_pkinase", "n": 200_000, "nlist": 40_000},
        # a long model's survivors
        {"name": "vit_m2400_3k", "kind": "vit", "model": "m2400_s1", "n": 20_000, "nlist": 3_000},
        # a database streamed from host memory, used once
        {"name": "host_m400_1m", "kind": "host", "M": 400, "n": 1_000_000, "lmax": 35000, "long_frac": 0.0},
        # hmmsearch's filter cascade with a Pfam model from host memory
        {"name": "filters_m260_300k", "kind": "filters", "model": "tut_pkinase", "n": 300_000, "block": 100_000},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["dropin", "search", "search", "search", "batch", "bias", "vit", "host", "filters"])
    if kind == "dropin":
        return {"kind": kind, "M": _log(rng, 20, 2400), "n": rng.randint(6, 32), "lmax": rng.choice([1000, 5000])}
    if kind in ("search", "host"):
        M = _log(rng, 20, 2400)
        long_frac = rng.choice([0.0, 0.0, 0.02])
        mean = MEAN_LEN + long_frac * 20000
        n = min(_log(rng, 2_000, 2_000_000 if kind == "search" else 1_000_000),
                int(MOST_CELLS / (2 if kind == "host" else 1) / M / mean))
        return {"kind": kind, "M": M, "n": n, "lmax": rng.choice([5000, 35000]), "long_frac": long_frac}
    if kind == "batch":
        return {"kind": kind, "nprof": rng.randint(5, 48), "n": _log(rng, 3_000, 40_000), "lmax": 35000}
    if kind == "filters":
        model = rng.choice(sorted(CASCADE))
        return {"kind": kind, "model": model, "n": _log(rng, 5_000, 300_000), "block": rng.choice([30_000, 100_000])}
    models = CASCADE if kind == "bias" else VITERBI
    model = rng.choice(sorted(models))
    nlist = min(_log(rng, 200, 40_000), int(40_000 * 400 / models[model]))
    return {"kind": kind, "model": model, "n": nlist * rng.randint(1, 5) + 7, "nlist": nlist}


# ---- inputs ------------------------------------------------------------------

_CTX = {}


def _ctx():
    """The program's one context."""
    if "ctx" not in _CTX:
        _CTX["ctx"] = api.Context(0)
    return _CTX["ctx"]


def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return g


def _sequences(seed, n, *, lmax, long_frac=0.0, emit=None, hom_frac=0.0, pinned=False):
    """n sequences as a SeqSet (codes in pinned memory if asked); hom_frac of
    them carry a stretch drawn from emit [M, 20]."""
    g = _gen(seed)
    dev = "cuda"
    lens = torch.exp(torch.randn(n, generator=g, device=dev, dtype=torch.float64) * 0.7 + math.log(300.0))
    lens = lens.round().clamp(10, lmax).to(torch.int64)
    if long_frac > 0:
        m = torch.rand(n, generator=g, device=dev) < long_frac
        lens = torch.where(m, torch.randint(5000, 35001, (n,), generator=g, device=dev), lens)
    off = torch.zeros(n + 1, dtype=torch.int64, device=dev)
    torch.cumsum(lens, 0, out=off[1:])
    total = int(off[-1])
    bg = F.AMINO_BG.astype(np.float64) / F.AMINO_BG.astype(np.float64).sum() * 0.995
    lut = np.searchsorted(np.cumsum(np.append(bg, 0.005)), (np.arange(65536) + 0.5) / 65536.0, side="right")
    lut = np.minimum(lut, 20)
    lut[lut == 20] = F.CODE_X
    lut = torch.from_numpy(lut.astype(np.uint8)).to(dev)
    codes = torch.empty(total, dtype=torch.uint8, device=dev)
    for a in range(0, total, 1 << 27):
        b = min(total, a + (1 << 27))
        codes[a:b] = lut[torch.randint(0, 65536, (b - a,), generator=g, device=dev, dtype=torch.int32).long()]
    nh = int(round(n * hom_frac))
    if nh and emit is not None:
        M = emit.shape[0]
        cdf = torch.from_numpy(np.cumsum(emit, axis=1)).to(dev)
        cdf = cdf / cdf[:, -1:]
        who = torch.randperm(n, generator=g, device=dev)[:nh]
        k0 = torch.randint(0, max(1, M // 3), (nh,), generator=g, device=dev)
        k1 = k0 + 1 + ((M - k0).double() * (0.5 + 0.5 * torch.rand(nh, generator=g, device=dev))).long()
        core = torch.minimum(torch.clamp(k1, max=M) - k0, lens[who])
        at = off[who] + ((lens[who] - core + 1).double() * torch.rand(nh, generator=g, device=dev).double()).long()
        which = torch.repeat_interleave(torch.arange(nh, device=dev), core)
        step = torch.arange(which.numel(), device=dev) - torch.repeat_interleave(torch.cumsum(core, 0) - core, core)
        r = torch.rand(which.numel(), generator=g, device=dev, dtype=torch.float64)
        new = (cdf[k0[which] + step] < r[:, None]).sum(1).clamp(max=19)
        codes[at[which] + step] = new.to(torch.uint8)
    if pinned:
        hc = torch.empty(total, dtype=torch.uint8, pin_memory=True)
        ho = torch.empty(n + 1, dtype=torch.int64, pin_memory=True)
        hc.copy_(codes)
        ho.copy_(off)
        return F.SeqSet(hc.numpy(), ho.numpy())
    return F.SeqSet(codes.cpu().numpy(), off.cpu().numpy())


def _vprofile(model):
    return F.read_vprofile(os.path.join(GOLDEN, "vit_%s.vprof" % model))


def _cascade(model):
    pipe = F.read_pipe(os.path.join(GOLDEN, "pipe_%s.pres" % model))
    own = os.path.join(GOLDEN, "pipe_%s.prof" % model)
    p = F.read_profile(own if os.path.exists(own) else os.path.join(GOLDEN, "%s.prof" % model))
    p.mmu, p.mlambda = pipe.mmu, pipe.mlambda
    return p, pipe


def _v_emission(v):
    """Match emissions from a ViterbiFilter profile's int16 scores."""
    k = np.arange(v.M)
    sc = v.rwv[:20, k % v.Q8, k // v.Q8].astype(np.float64).T / v.scale_w
    e = F.AMINO_BG[None, :].astype(np.float64) * np.exp(sc)
    return e / e.sum(1, keepdims=True)


def _list(seed, n, nlist):
    """A survivor list: nlist of n sequences, ascending."""
    return np.sort(np.random.default_rng(seed).choice(n, size=nlist, replace=False)).astype(np.int64)


def prepare(case, seed):
    kind = case["kind"]
    ctx = _ctx()
    if kind == "dropin":
        p = api.sample_profile(case["M"], 1 + seed % 1000)
        s = _sequences(seed, case["n"], lmax=case["lmax"], emit=F.emission_probs(p), hom_frac=0.1)
        dsq = [np.concatenate([[255], s.seq(i), [255]]).astype(np.uint8) for i in range(s.n)]
        return {"case": case, "ctx": ctx, "p": p, "dsq": dsq, "tjb": [api.tjb_b(p.scale_b, len(d) - 2) for d in dsq]}
    if kind in ("search", "host"):
        p = api.sample_profile(case["M"], 1 + seed % 1000, ctx)
        s = _sequences(seed, case["n"], lmax=case["lmax"], long_frac=case["long_frac"], emit=F.emission_probs(p),
                       hom_frac=0.02, pinned=kind == "host")
        st = {"case": case, "ctx": ctx, "prof": api.DeviceProfile(ctx, p)}
        if kind == "host":
            out = torch.empty((2, s.n), dtype=torch.uint8, pin_memory=True)
            return dict(st, seqs=s, out=out, np_out=(out[0].numpy(), out[1].numpy()))
        return dict(st, db=api.DeviceDB(ctx, s), out=torch.empty((2, s.n), dtype=torch.uint8, device="cuda"))
    if kind == "batch":
        Ms = np.random.default_rng(seed).integers(50, 1501, size=case["nprof"])
        profs = [api.sample_profile(int(M), 1 + i + seed % 1000, ctx) for i, M in enumerate(Ms)]
        s = _sequences(seed, case["n"], lmax=case["lmax"], emit=F.emission_probs(profs[0]), hom_frac=0.01)
        db = api.DeviceDB(ctx, s)
        out = torch.empty((2, case["nprof"], s.n), dtype=torch.uint8, device="cuda")
        batch = api.Batch(ctx, profs, db, out[0].data_ptr(), out[1].data_ptr())
        return {"case": case, "ctx": ctx, "db": db, "batch": batch, "out": out}
    if kind == "bias":
        p, pipe = _cascade(case["model"])
        s = _sequences(seed, case["n"], lmax=35000, emit=F.emission_probs(p), hom_frac=0.1)
        return {"case": case, "ctx": ctx, "db": api.DeviceDB(ctx, s), "ids": _list(seed, s.n, case["nlist"]),
                "compo": pipe.compo, "M": p.M, "seqs": s}
    if kind == "vit":
        v = _vprofile(case["model"])
        s = _sequences(seed, case["n"], lmax=35000, emit=_v_emission(v), hom_frac=0.1)
        return {"case": case, "ctx": ctx, "db": api.DeviceDB(ctx, s), "ids": _list(seed, s.n, case["nlist"]),
                "vprof": api.DeviceVProfile(ctx, v), "v": v, "seqs": s}
    p, pipe = _cascade(case["model"])
    s = _sequences(seed, case["n"], lmax=35000, emit=F.emission_probs(p), hom_frac=0.02, pinned=True)
    return {"case": case, "ctx": ctx, "p": p, "pipe": pipe, "v": _vprofile(case["model"]), "seqs": s}


def run(state):
    case = state["case"]
    kind, ctx = case["kind"], state["ctx"]
    if kind == "dropin":
        got = [ctx.MSVFilter(d, len(d) - 2, state["p"], t) for d, t in zip(state["dsq"], state["tjb"])]
        return {"status": np.array([g[0] for g in got], np.int32), "sc": np.array([g[1] for g in got], np.float32)}
    if kind == "search":
        out = state["out"]
        api.search_device(ctx, state["prof"], state["db"], out[0].data_ptr(), out[1].data_ptr())
        return {"xj": out[0], "flags": out[1]}
    if kind == "batch":
        state["batch"].run()
        return {"xj": state["out"][0], "flags": state["out"][1]}
    if kind == "bias":
        return {"sc": api.biasfilter(ctx, state["compo"], state["M"], state["db"], state["ids"])}
    if kind == "vit":
        status, sc = api.vitfilter(ctx, state["vprof"], state["db"], state["ids"])
        return {"status": status, "sc": sc}
    if kind == "host":
        xj, flags = api.search_host(ctx, state["prof"], state["seqs"], out=state["np_out"])
        return {"xj": xj, "flags": flags}
    pipe = state["pipe"]
    hits, stats = api.pipeline_filters(ctx, state["p"], state["seqs"], vprof=state["v"], compo=pipe.compo, vmu=pipe.vmu,
                                       vlambda=pipe.vlambda, block_size=case["block"])
    # per sequence, as a program that joins the hits to its own tables keeps them
    n, at = state["seqs"].n, hits["seq_index"]
    out = {k: np.full(n, np.nan, np.float32) for k in ("usc", "nullsc", "filtersc", "vfsc")}
    for k, v in out.items():
        v[at] = hits[k]
    out["hit"] = np.zeros(n, np.uint8)
    out["hit"][at] = 1
    out["past"] = np.array([stats.n_past_msv, stats.n_past_bias, stats.n_past_vit], np.int64)
    return out


def work(case):
    """Residues read once, results written once; per DP cell one add and two
    maxima (the cell's floor and the running maximum) for MSV, 4 candidates for
    a match cell, 2 for an insert and 2 for a delete cell (add and maximum each)
    and the emission for the ViterbiFilter; per residue of the bias filter 4
    multiplies by transitions, 2 by emissions, 2 adds, 2 divisions and a log."""
    kind = case["kind"]
    n = case["nlist"] if kind in ("bias", "vit") else case["n"]
    res = n * (MEAN_LEN + 20000.0 * case.get("long_frac", 0.0))
    if kind in ("dropin", "search", "host"):
        return {"bytes": res + 2 * n + 29 * case["M"], "flops": 3.0 * case["M"] * res}
    if kind == "batch":
        return {"bytes": res + case["nprof"] * (2 * n + 29 * 775), "flops": 3.0 * 775 * case["nprof"] * res}
    if kind == "bias":
        return {"bytes": res + 4 * n, "flops": 11.0 * res}
    if kind == "vit":
        M = VITERBI[case["model"]]
        return {"bytes": res + 5 * n + 2 * 37 * M, "flops": 18.0 * M * res}
    M = CASCADE[case["model"]]
    past = 0.04                          # sequences past MSV: 2% by chance, 2% homologs
    return {"bytes": res + 24 * past * n, "flops": (3.0 * M + past * (11.0 + 18.0 * M)) * res}


# ---- 64-bit results -----------------------------------------------------------

def _by_length(seqs, ids):
    """Sequences longest first: their order and an accessor of row i's codes and live count."""
    lens = seqs.lengths[ids]
    order = np.argsort(-lens, kind="stable")
    lens = lens[order]
    start = torch.from_numpy(np.ascontiguousarray(seqs.off[ids[order]])).cuda()
    codes = torch.from_numpy(seqs.codes).cuda()
    return order, lens, lambda i, m: codes[start[:m] + i].long()


def _exact_msv(p, body, tjb):
    """p7_MSVFilter's score of one sequence: integer dynamic programming."""
    costs = p.node_costs().astype(np.int64)
    tjbm = tjb + p.tbm_b
    xJ, xB = 0, max(p.base_b - tjbm, 0)
    dp = np.zeros(p.M + 1, np.int64)
    for x in body:
        prev = np.maximum(dp[:-1], xB)
        dp[1:] = np.maximum(np.minimum(prev + p.bias_b, 255) - costs[x], 0)
        xE = int(dp.max())
        if xE + p.bias_b >= 255:
            return math.inf
        xJ = max(xJ, xE - p.tec_b)
        xB = max(max(p.base_b, xJ) - tjbm, 0)
    return (float(xJ - tjb) - p.base_b) / p.scale_b - 3.0


def _exact_bias(state):
    """Two-state Forward score of the filter model in 64 bits."""
    seqs, ids, M = state["seqs"], state["ids"], state["M"]
    bg = F.AMINO_BG.astype(np.float64)
    eo = np.ones((29, 2))
    eo[:20, 1] = state["compo"].astype(np.float64) / bg
    sets = {21: (2, 11), 22: (7, 9), 23: (3, 13), 24: (8,), 25: (1,), 26: tuple(range(20))}
    for x, ys in sets.items():
        eo[x, 1] = state["compo"].astype(np.float64)[list(ys)].sum() / bg[list(ys)].sum()
    eo = torch.from_numpy(eo).cuda()
    order, lens, row = _by_length(seqs, ids)
    L = torch.from_numpy(lens).cuda().double()
    p1 = L / (L + 1)
    l1 = M / 8.0
    t10, t11 = 1 / (l1 + 1), l1 / (l1 + 1)
    d = torch.zeros((len(ids), 2), dtype=torch.float64, device="cuda")
    lsc = torch.zeros(len(ids), dtype=torch.float64, device="cuda")
    for i in range(int(lens[0])):
        m = int(np.searchsorted(-lens, -i, side="left"))            # lens > i
        e = eo[row(i, m)]
        if i == 0:
            nd = e * torch.tensor([0.999, 0.001], dtype=torch.float64, device="cuda")
        else:
            a, b = d[:m, 0], d[:m, 1]
            nd = torch.stack([a * p1[:m] + b * t10, a * (1 - p1[:m]) + b * t11], 1) * e
        mx = nd.max(1).values
        d[:m] = nd / mx[:, None]
        lsc[:m] += mx.log()
    sc = lsc + d.sum(1).log() + L * p1.log() + (1 - p1).log()
    out = np.empty(len(ids))
    out[order] = sc.cpu().numpy()
    return out


def _exact_vit(state):
    """p7_ViterbiFilter's score: the integer recurrence with every delete path."""
    v, seqs, ids = state["v"], state["seqs"], state["ids"]
    M, Q8, FLOOR = v.M, v.Q8, -32768
    k = np.arange(M)
    tr = v.twv[:7 * Q8].reshape(Q8, 7, 8).astype(np.int32)[k % Q8, :, k // Q8]           # [M, 7]
    bm, mm, im, dm, md, mi, ii = [torch.from_numpy(np.ascontiguousarray(tr[:, j])).cuda() for j in range(7)]
    dd = v.twv[7 * Q8:].astype(np.int32)[k % Q8, k // Q8]                                # out of node k
    dcum = np.concatenate([[0], np.cumsum(dd[:-1].astype(np.int64))])                    # node 1 .. M
    dcum = torch.from_numpy(dcum.astype(np.int32)).cuda()
    em = torch.from_numpy(np.ascontiguousarray(v.rwv[:, k % Q8, k // Q8].astype(np.int32))).cuda()
    order, lens, row = _by_length(seqs, ids)
    n = len(ids)
    move = np.array([api.lib().msvgb_vit_move_cost(v.scale_w, v.nj, int(x)) for x in lens], np.int32)
    mv = torch.from_numpy(move).cuda()
    full = lambda: torch.full((n, M), FLOOR, dtype=torch.int32, device="cuda")  # noqa: E731
    Mm, Im, Dm = full(), full(), full()
    xC = torch.full((n,), FLOOR, dtype=torch.int32, device="cuda")
    xJ, xN = xC.clone(), torch.full_like(xC, v.base_w)
    xB = xN + mv
    over = torch.zeros(n, dtype=torch.bool, device="cuda")
    shift = lambda t: torch.nn.functional.pad(t[:, :-1], (1, 0), value=FLOOR)  # noqa: E731
    for i in range(int(lens[0])):
        m = int(np.searchsorted(-lens, -i, side="left"))
        A, I, D = Mm[:m], Im[:m], Dm[:m]
        s = torch.maximum(torch.maximum(shift(A) + mm, shift(I) + im), torch.maximum(shift(D) + dm, xB[:m, None] + bm))
        s = (s.clamp(min=FLOOR) + em[row(i, m)]).clamp(FLOOR, 32767)
        Im[:m] = torch.maximum(A + mi, I + ii).clamp(min=FLOOR)
        Mm[:m] = s
        D = shift((s + md).clamp(min=FLOOR))
        Dm[:m] = (torch.cummax(D - dcum, 1).values + dcum).clamp(min=FLOOR)
        xE = s.max(1).values
        over[:m] |= xE >= 32767
        xN[:m] += int(v.xw[1][1])
        xC[:m] = torch.maximum(xC[:m] + int(v.xw[3][1]), xE + int(v.xw[0][0]))
        xJ[:m] = torch.maximum(xJ[:m] + int(v.xw[2][1]), xE + int(v.xw[0][1]))
        xB[:m] = torch.maximum(xJ[:m], xN[:m]) + mv[:m]
    sc = (xC.double() + mv.double() - v.base_w) / v.scale_w - 3.0
    sc = torch.where(over, math.inf, torch.where(xC <= FLOOR, -math.inf, sc))
    out = np.empty(n)
    out[order] = sc.cpu().numpy()
    return out


def exact(case, seed):
    kind = case["kind"]
    if kind == "dropin":
        st = prepare(case, seed)
        return {"status": None, "sc": np.array([_exact_msv(st["p"], d[1:-1], t) for d, t in zip(st["dsq"], st["tjb"])])}
    if kind == "bias":
        return {"sc": _exact_bias(prepare(case, seed))}
    if kind == "vit" and case["nlist"] * VITERBI[case["model"]] <= 12_000_000:
        return {"status": None, "sc": _exact_vit(prepare(case, seed))}
    return None
