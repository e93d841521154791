"""Performance cases: what a program has this engine do, through its public entry points.

A case is a dict of plain values; `kind` says which entry points it goes through:

  job       Engine.init / step / population: one whole design run of G generations
  batch     Batch.step over many proteins at once, then every member's population
  evaluate  Engine.evaluate: objectives of solutions the caller holds on the host
  mutate    Engine.mutate: one variation step on the caller's parents
  select    Engine.select: one environmental selection on the caller's objectives
  stem      hairpin_noalloc: stem objective of device-resident nucleotides

Inputs come from the seed alone and are made with numpy, so `exact` can restate what
the evaluators should return in 64 bits without the engine.
"""
import importlib
import math

import numpy as np
import torch

pe = importlib.import_module("protein_encoding_v2_nsga-iii_b200")

# the standard genetic code, codons grouped by amino acid (index order ACDEFGHIKLMNPQRSTVWY, stop)
CODE = ("GCU GCC GCA GCG|UGU UGC|GAU GAC|GAA GAG|UUU UUC|GGU GGC GGA GGG|CAU CAC|AUU AUC AUA|AAA AAG|"
        "UUA UUG CUU CUC CUA CUG|AUG|AAU AAC|CCU CCC CCA CCG|CAA CAG|CGU CGC CGA CGG AGA AGG|"
        "UCU UCC UCA UCG AGU AGC|ACU ACC ACA ACG|GUU GUC GUA GUG|UGG|UAU UAC|UAA UAG UGA")
STOP = 20


def listed():
    return [
        # the smallest design run: a short protein, two CDSs; launches and latency count
        dict(name="job_small", kind="job", L=200, m=2, N=128, G=100, pm=0.05, p=6, objectives=1, gc=0, string=0,
             protein="uniform", progress=False),
        # the ordinary design run, 500 generations, the objectives of every generation
        # read behind it as a program that shows progress does
        dict(name="job_1000", kind="job", L=1000, m=8, N=1024, G=500, pm=0.02, p=8, objectives=1, gc=0, string=0,
             protein="uniform", progress=True),
        # the same with the full set of six objectives and its many more reference points
        dict(name="job_1000_six", kind="job", L=1000, m=8, N=1024, G=500, pm=0.02, p=0, objectives=0, gc=0, string=0,
             protein="uniform", progress=False),
        # a long protein and a large population
        dict(name="job_3000", kind="job", L=3000, m=4, N=4096, G=200, pm=0.02, p=0, objectives=1, gc=0, string=0,
             protein="uniform", progress=False),
        # the same with the longest repeated or common substring as the string objective
        dict(name="job_3000_lrcs", kind="job", L=3000, m=4, N=4096, G=200, pm=0.02, p=0, objectives=1, gc=0, string=1,
             protein="uniform", progress=False),
        # the longest proteins that are designed (the upper end of the served mix)
        dict(name="job_5000", kind="job", L=5000, m=6, N=1024, G=100, pm=0.02, p=0, objectives=1, gc=1, string=0,
             protein="uniform", progress=False),
        # a protein of tandem repeats (elastin, silk, collagen): the one whose designs are
        # hardest to keep free of stems and repeats
        dict(name="job_repeat", kind="job", L=601, m=5, N=500, G=100, pm=0.02, p=0, objectives=1, gc=0, string=0,
             protein="repeat", progress=False),
        # many proteins at once, L log-uniform in [100, 3000], m in {2, 4, 8}
        dict(name="batch_32", kind="batch", jobs=32, L=100, Lmax=3000, N=512, G=300, pm=0.02, string=0,
             queue=False),
        # scoring a set of solutions that another program made
        dict(name="evaluate_1000", kind="evaluate", L=1000, m=8, N=1024, objectives=0, gc=0, string=0,
             protein="uniform"),
        # one variation step on solutions that another program keeps
        dict(name="mutate_1000", kind="mutate", L=1000, m=8, N=1024, pm=0.02, objectives=1, gc=0, string=0),
        # one environmental selection for a program with its own objectives
        dict(name="select_4096", kind="select", N=4096, objectives=1, p=0),
        # the stem objective of solutions that are on the device already
        dict(name="stem_1000", kind="stem", L=1000, m=8, N=1024),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


# stem or substring cells of one generation, about: what bounds a drawn run's length
def _cells(m, L, N, string):
    pairs = m * (m + 1) / 2 if string else m
    return 0.3 * N * pairs * (3 * L) ** 2 / (1 if string else 2)


def draw(rng):
    kind = rng.choice(["job", "job", "job", "job", "batch", "evaluate", "mutate", "select", "stem"])
    if kind == "job":
        L, m, N = _log(rng, 50, 5000), rng.randint(2, 10), _log(rng, 64, 4096)
        string = int(rng.random() < 0.25)
        protein = "repeat" if rng.random() < 0.2 else "uniform"
        G = _log(rng, 50, 500)
        # no more than the longest listed run: generations x population, and cells
        most = 1.5e13 if protein == "uniform" else 1e12
        G = max(2, min(G, int(8e5 / N), int(most / _cells(m, L, N, string))))
        while _cells(m, L, N, string) * G > most and N > 64:
            N = max(64, N // 2)
        return dict(kind=kind, L=L, m=m, N=N, G=G, pm=rng.choice([0.01, 0.02, 0.05]), p=0,
                    objectives=rng.choice([0, 1, 1]), gc=rng.choice([0, 0, 1]), string=string, protein=protein,
                    progress=rng.random() < 0.3)
    if kind == "batch":
        lo = _log(rng, 50, 500)
        jobs, N, G = rng.randint(3, 32), _log(rng, 64, 512), _log(rng, 20, 200)
        return dict(kind=kind, jobs=jobs, L=lo, Lmax=_log(rng, lo, 2500), N=N, G=G, pm=0.02,
                    string=int(rng.random() < 0.2), queue=rng.random() < 0.3)
    if kind == "select":
        six = rng.random() < 0.4
        return dict(kind=kind, N=_log(rng, 32, 4096), objectives=0 if six else 1, p=0)
    if kind == "stem":
        L, m = _log(rng, 20, 4000), rng.randint(1, 10)
        most = int(7.5e6 / (m * (0.76 * L + 40)))  # the call's fixed scratch
        return dict(kind=kind, L=L, m=m, N=max(1, min(_log(rng, 1, 2000), most)))
    L, m = _log(rng, 50, 3000), rng.randint(2, 10)
    N = max(1, min(_log(rng, 1, 1024), int(1.6e7 / (m * L))))
    c = dict(kind=kind, L=L, m=m, N=N, objectives=rng.choice([0, 1]), gc=rng.choice([0, 1]),
             string=int(rng.random() < 0.25))
    if kind == "mutate":
        c["pm"] = rng.choice([0.01, 0.02, 0.05])
    else:
        c["protein"] = "repeat" if rng.random() < 0.3 else "uniform"
        if c["protein"] == "repeat":
            c["N"] = max(1, min(c["N"], int(4e10 / _cells(m, L, 1, c["string"]))))
    return c


# ------------------------------------------------------------------- inputs


def _table(rng):
    """The standard code, Dirichlet(1) weights scaled to a largest of 1 per amino acid,
    each amino acid's codons in ascending weight; uniform codon-pair scores."""
    nt, weight, start, count = [], [], [], []
    for group in CODE.split("|"):
        codons = group.split()
        w = rng.exponential(size=len(codons))
        w = (w / w.max()).astype(np.float32)
        order = np.argsort(w, kind="stable")
        start.append(len(nt))
        count.append(len(codons))
        nt += [["ACGU".index(x) for x in codons[i]] for i in order]
        weight += [w[i] for i in order]
    cps = rng.uniform(-0.4, 0.4, 61 * 61).astype(np.float32)
    return dict(nt=np.array(nt, np.uint8), weight=np.array(weight, np.float32), cps=cps,
                start=np.array(start, np.int8), count=np.array(count, np.int8), ref_gc3=float(np.float32(0.3810)),
                ref_gc=float(np.float32(0.3977)))


def _protein(rng, L, kind):
    """L amino acids and the stop: uniform over the 20, or a motif of 4 to 8 residues
    repeated, one residue in 20 replaced."""
    aa = rng.integers(0, 20, L)
    if kind == "repeat":
        motif = rng.integers(0, 20, int(rng.integers(4, 9)))
        aa = np.where(rng.random(L) < 0.05, aa, np.resize(motif, L))
    return np.append(aa, STOP).astype(np.int8)


def _codons(rng, aa, table, N, m):
    """N solutions of m CDSs: a uniformly drawn synonym at every position."""
    k = table["count"][aa].astype(np.float32)
    pick = (rng.random((N, m, len(aa)), dtype=np.float32) * k).astype(np.uint8)
    return table["start"][aa].astype(np.uint8) + np.minimum(pick, (k - 1).astype(np.uint8))


def _solutions(case, seed):
    rng = np.random.default_rng(seed)
    table = _table(rng)
    aa = _protein(rng, case["L"], case.get("protein", "uniform"))
    return aa, table, _codons(rng, aa, table, case["N"], case["m"])


def _objectives(case, seed):
    """Objectives of 2N solutions as a running design holds them (minimised): a codon
    adaptation that trades against the distance of the CDSs, counts over the length, a
    stem of a few more pairs than the shortest; the first half, the parents, further on."""
    rng = np.random.default_rng(seed)
    n2, L = 2 * case["N"], 501
    behind = np.where(np.arange(n2) < case["N"], 0.0, np.abs(rng.normal(0, 0.03, n2)))
    cai = 0.55 + 0.4 * rng.random(n2)
    hd = 0.33 * np.sqrt(1.0 - cai ** 2) + rng.normal(0, 0.01, n2)
    gc = np.abs(rng.normal(0.0, 0.06, n2)) + 0.1 * np.abs(cai - 0.8)
    sl = 9 + rng.poisson(1.5, n2)
    cols = [-(cai - behind), -np.round((hd - behind) * 3 * L) / (3 * L), np.round((gc + behind) * L) / L,
            sl / ((3 * L - 4) // 2)]
    if case["objectives"] == 0:
        cols[1:1] = [0.2 - 0.5 * rng.random(n2) * (1 - behind), -rng.poisson(40, n2) / (L - 1)]
    obj = np.stack(cols, axis=1).astype(np.float32)
    return obj, obj[rng.integers(0, n2, obj.shape[1])]


def _engine(case, aa, table, seed, m=None):
    return pe.Engine(aa, pe.CodonTable.from_arrays(table), m or case["m"], case["N"], case.get("pm", 0.02),
                     objectives=case.get("objectives", 1), gc_mode=case.get("gc", 0), ref_p=case.get("p", 0),
                     seed=seed, sl_kind=case.get("string", 0))


def _member(case, j):
    """Length and CDSs of a batch's protein j: lengths log-uniform (a golden-ratio
    sequence), m in {2, 4, 8}."""
    u = (0.5 + j * 0.6180339887498949) % 1.0
    return int(round(case["L"] * (case["Lmax"] / case["L"]) ** u)), (2, 4, 8)[(j + j // 3) % 3]


def _scorer(case, aa, table, seed):
    """An engine that scores or varies a caller's solutions; its own population is small."""
    return _engine(dict(case, N=64), aa, table, seed)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "job":
        rng = np.random.default_rng(seed)
        table = _table(rng)
        eng = _engine(case, _protein(rng, case["L"], case["protein"]), table, seed)
        s = dict(case=case, eng=eng)
        if case["progress"]:
            s["ring"] = [torch.empty((2 * eng.N, eng.M), dtype=torch.float32, pin_memory=True) for _ in range(2)]
        return s
    if kind == "batch":
        rng = np.random.default_rng(seed)
        engines = []
        for j in range(case["jobs"]):
            table = _table(rng)
            L, m = _member(case, j)
            engines.append(_engine(case, _protein(rng, L, "uniform"), table, seed + j, m=m))
            engines[-1].init()
        batch = pe.Batch(engines)
        batch.set_scan_queue(case["queue"])
        return dict(case=case, engines=engines, batch=batch)
    if kind == "select":
        obj, ext = _objectives(case, seed)
        rng = np.random.default_rng(seed)
        table = _table(rng)
        eng = _engine(dict(case, m=2), _protein(rng, 30, "uniform"), table, seed)
        return dict(case=case, eng=eng, obj=obj, ext=ext)
    aa, table, ids = _solutions(case, seed)
    if kind == "stem":
        dev = torch.device("cuda", torch.cuda.current_device())
        n, m = ids.shape[:2]
        nt = torch.from_numpy(table["nt"]).to(dev)[torch.from_numpy(ids).to(dev).long()].reshape(n, m, -1).contiguous()
        return dict(case=case, nt=nt, value=torch.empty(n, device=dev),
                    pql=torch.empty((n, 3), dtype=torch.int32, device=dev),
                    cds=torch.empty(n, dtype=torch.int8, device=dev))
    eng = _scorer(case, aa, table, seed)
    s = dict(case=case, eng=eng, ids=ids)
    if kind == "mutate":
        s["scores"] = eng.evaluate(ids)
        s["idx"] = np.arange(case["N"], dtype=np.int32)
        s["generation"] = seed % 1000
    return s


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "job":
        eng = state["eng"]
        eng.init()
        if case["progress"]:
            ring = state["ring"]
            for g in range(case["G"]):
                eng.step(1)
                eng.read_objectives_async(ring[g & 1].data_ptr())
        else:
            eng.step(case["G"])
        return eng.population()
    if kind == "batch":
        for e in state["engines"]:
            e.init()
        state["batch"].step(case["G"])
        state["batch"].synchronize()
        ids, *rest = zip(*(e.population() for e in state["engines"]))
        return [list(ids), [np.concatenate(x) for x in rest]]
    if kind == "evaluate":
        return state["eng"].evaluate(state["ids"])
    if kind == "mutate":
        return state["eng"].mutate(state["generation"], state["idx"], state["ids"], *state["scores"])
    if kind == "select":
        eng = state["eng"]
        surv, front, ext, info = eng.select(5, state["obj"], state["ext"])
        whole = np.array([info.rank_count, info.last_front_size, info.n_fronts, info.cut, info.hyp_exception])
        return [surv, front, ext, whole] + [np.array(v[: eng.M], np.float32) for v in (info.ideal, info.worst, info.nadir)]
    nt = state["nt"]
    pe.hairpin_noalloc(nt.data_ptr(), nt.shape[0], nt.shape[1], nt.shape[2] // 3, state["value"].data_ptr(),
                       state["pql"].data_ptr(), state["cds"].data_ptr(), torch.cuda.current_stream().cuda_stream)
    return [state["value"], state["pql"], state["cds"]]


# ---------------------------------------------------------------------- work


def _points(M, N, p):
    if p <= 0:  # the largest p whose points do not outnumber the population
        p = 1
        while math.comb(M + p, p + 1) <= N:
            p += 1
    return math.comb(M + p - 1, p)


def _light(N, m, L):  # one look at every codon (CAI, GC) and at every pair of CDSs by plane words (HD)
    return N * (3 * m * L + m * (m - 1) / 2 * L / 2)


def _string(N, m, L, string):  # one word of each sequence entered in a table and looked up
    return 20 * N * (m * (m + 1) / 2 if string else m) * 3 * L


def _select(N, M, R):  # every pair compared, every solution's distance to every point
    return 2 * M * (2 * N) ** 2 + 7 * M * 2 * N * R


def _generation(m, L, N, M, R, string):
    """A generation: the parents' codons read, the children's written, the objectives of
    both; one operator in five redraws every CDS, the others one."""
    share = (m + 4) / 5 / m
    by = 2 * N * m * L + 2 * N * M * 4 * 2
    return by, share * (_light(N, m, L) + _string(N, m, L, string)) + 8 * N * share * m * L + _select(N, M, R)


def work(case):
    kind, N = case["kind"], case["N"]
    M = 4 if case.get("objectives", 1) == 1 else 6
    if kind == "select":
        R = _points(M, N, case["p"])
        return dict(bytes=4 * M * (2 * N + R) + 12 * N, flops=_select(N, M, R))
    if kind == "batch":
        total = np.zeros(2)
        for L, m in (_member(case, j) for j in range(case["jobs"])):
            by, fl = _generation(m, L + 1, N, 4, _points(4, N, 0), case["string"])
            total += case["G"] * by + 2 * N * m * (L + 1), case["G"] * fl
        return dict(bytes=float(total[0]), flops=float(total[1]))
    m, L = case["m"], case["L"] + 1
    if kind == "job":
        by, fl = _generation(m, L, N, M, _points(M, N, case["p"]), case["string"])
        return dict(bytes=case["G"] * by + 2 * N * m * L,
                    flops=case["G"] * fl + _light(N, m, L) + _string(N, m, L, case["string"]))
    if kind == "mutate":
        return dict(bytes=2 * N * m * L, flops=8 * N * (m + 4) / 5 * L)
    if kind == "stem":
        L = case["L"] + 1
        return dict(bytes=N * m * 3 * L + 17 * N, flops=_string(N, m, L, 0))
    return dict(bytes=N * (m * L + 6 * M + 12), flops=_light(N, m, L) + _string(N, m, L, case["string"]))


# --------------------------------------------------------------------- exact


def _longest(eq, step):
    """Longest run of set cells along (r + 1, c + step) in every matrix of a batch."""
    best = torch.zeros(eq.shape[0], dtype=torch.int64, device=eq.device)
    cur, k = eq, 0
    while True:
        any_ = cur.flatten(1).any(1)
        if not bool(any_.any()):
            return best
        k += 1
        best[any_] = k
        if cur.shape[1] < 2 or cur.shape[2] < 2:
            return best
        cur = (eq[:, : cur.shape[1] - 1, k:] if step < 0 else eq[:, : cur.shape[1] - 1, : cur.shape[2] - 1]) & (
            cur[:, 1:, :-1] if step < 0 else cur[:, 1:, 1:])


def _stems(nt):
    """Longest stem of every sequence: pairs (r, c), (r + 1, c - 1), .. with c - r >= 5."""
    n = nt.shape[-1]
    flat = nt.reshape(-1, n)
    r = torch.arange(n, device=nt.device)
    loop = r[None, :] - r[:, None] >= 5
    out = []
    for x in torch.split(flat, max(1, int(2e8 / n ** 2))):
        out.append(_longest(((x[:, :, None] + x[:, None, :]) == 3) & loop, -1))
    return torch.cat(out).reshape(nt.shape[:-1])


def _substrings(nt):
    """Longest run shared by two CDSs of a solution, or repeated in one."""
    n, m = nt.shape[-1], nt.shape[1]
    r = torch.arange(n, device=nt.device)
    later = r[None, :] > r[:, None]
    best = torch.zeros(nt.shape[0], dtype=torch.int64, device=nt.device)
    for a in range(m):
        for b in range(a, m):
            got = []
            size = max(1, int(2e8 / n ** 2))
            for x, y in zip(torch.split(nt[:, a], size), torch.split(nt[:, b], size)):
                eq = x[:, :, None] == y[:, None, :]
                got.append(_longest(eq & later if a == b else eq, 1))
            best = torch.maximum(best, torch.cat(got))
    return best


def exact(case, seed):
    kind = case["kind"]
    if kind == "select":  # ideal and worst points; the others follow from comparisons alone
        obj = _objectives(case, seed)[0].astype(np.float64)
        return [None, None, None, None, obj.min(0), obj.max(0), None]
    if kind not in ("evaluate", "stem"):
        return None  # whole runs: whole numbers, and objectives that `evaluate` covers
    N, m, n = case["N"], case["m"], 3 * (case["L"] + 1)
    if N * (m * (m + 1) / 2 if case.get("string") else m) * n ** 2 > 4e11:
        return None
    dev = torch.device("cuda") if torch.cuda.is_available() else torch.device("cpu")
    aa, table, ids = _solutions(case, seed)
    nt = torch.from_numpy(table["nt"][ids].reshape(N, m, n)).to(dev)
    if kind == "stem":
        return [(_stems(nt).max(1).values.double() / ((n - 4) // 2)).cpu(), None, None]
    i = ids.astype(np.int64)
    L = ids.shape[2]
    with np.errstate(divide="ignore"):
        cai = np.exp(np.log(table["weight"].astype(np.float64))[i].mean(2)).min(1)
    seqs = table["nt"][ids].reshape(N, m, n)
    hd = np.min([(seqs[:, a] != seqs[:, b]).mean(1) for a in range(m) for b in range(a + 1, m)], axis=0)
    gcnt = (table["nt"] == 1) | (table["nt"] == 2)
    if case["gc"] == 0:
        gc = np.abs(gcnt[:, 2][i].mean(2) - table["ref_gc3"]).max(1)
    else:
        ref = n * table["ref_gc"]
        gc = (np.abs(gcnt.sum(1)[i].sum(2) - ref) / ref).max(1)
    sl = (_substrings(nt) / n if case["string"] else _stems(nt).max(1).values / ((n - 4) // 2)).double().cpu().numpy()
    cols = [-cai, -hd, gc, sl]
    if case["objectives"] == 0:
        pair = np.zeros((64, 64))
        pair[:61, :61] = table["cps"].astype(np.float64).reshape(61, 61)
        cbp = (pair[i[:, :, : L - 2], i[:, :, 1 : L - 1]].sum(2) / (L - 2)).min(1)
        t = table["nt"]
        stops = {tuple(t[c]) for c in (61, 62, 63)}
        hidden = np.array([[((t[x][1], t[x][2], t[y][0]) in stops) + ((t[x][2], t[y][0], t[y][1]) in stops)
                            for y in range(64)] for x in range(64)])
        hsc = (hidden[i[:, :, :-1], i[:, :, 1:]].sum(2) / (L - 1)).min(1)
        cols[1:1] = [-cbp, -hsc]
    return [np.stack(cols, 1), None, None]
