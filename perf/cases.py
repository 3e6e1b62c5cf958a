"""What users of this framework run, as measurable cases.

A case is one call that a program makes through the public entry points:
``run_l2`` on a resident panel (exact INT8 form, f64 form, CountSketch form,
with or without annotations, --keep and --extract), ``l2_from_bed_bytes`` on a
host file image, and the regressions (h2, rg, partitioned h2) on a server's
resident arrays or on host arrays.  Panels are seeded founder mosaics: each
haplotype copies one of F founders over segments of SEG SNPs, a share of the
genotypes is missing.
"""
from __future__ import annotations

import math

import numpy as np
import torch

SEG = 100          # SNPs a haplotype copies one founder for
FOUNDERS = 64
_kept = {}         # what a program keeps for its whole life: the context, the server


def listed():
    return [
        # a serving request for one small region of a resident 1000G-size panel: latency
        dict(name="region-int8", kind="l2", n=2490, m=1013, chroms=1, per_cm=266, form="int8", masked=True),
        # one chromosome through run_l2's defaults: f64 form, chunks of 200, 1 cM
        dict(name="chrom-fp64", kind="l2", n=2490, m=18627, chroms=1, per_cm=266, form="fp64", masked=False),
        # biobank: the largest exact run, per-SNP masking
        dict(name="biobank-int8", kind="l2", n=50000, m=100000, chroms=1, per_cm=1000, form="int8", masked=True),
        # a cohort subset on array SNPs: --keep and --extract, kb windows, chunks of 200, odd sizes
        dict(name="keep-extract-int8", kind="l2", n=20011, m=50021, chroms=3, per_cm=400, form="int8",
             masked=False, window="kb", keep=15003, extract=True),
        # partitioned LD scores: 97 resident annotations, l2 left on the device
        dict(name="partitioned-k97", kind="l2", n=10000, m=100000, chroms=5, per_cm=143, form="int8",
             masked=False, K=97, on_device=True),
        # CountSketch on a biobank panel, a small and a large d, and the MAF-aware form
        dict(name="sketch-d200", kind="l2", n=100000, m=50000, chroms=1, per_cm=1333, form="sketch", d=200,
             masked=True),
        dict(name="sketch-d1000-maf", kind="l2", n=20000, m=60007, chroms=2, per_cm=343, form="sketch", d=1000,
             maf_aware=True, masked=True),
        dict(name="sketch-d5000", kind="l2", n=100000, m=20011, chroms=1, per_cm=1333, form="sketch", d=5000,
             masked=True),
        # a whole .bed image in pinned host memory: validate, upload, compute, read back
        dict(name="bed-file-int8", kind="bed", n=50000, m=20011, chroms=1, per_cm=1000, form="int8", masked=True),
        # regressions on a server's resident arrays: h2 over 1,000 traits, 200 trait pairs, 97 annotations
        dict(name="h2-1000-traits", kind="h2", m=200000, traits=1000, blocks=200, lambda_gc=True),
        dict(name="rg-200-pairs", kind="rg", m=200000, traits=200, blocks=200),
        dict(name="h2-partitioned-k97", kind="h2p", m=300007, traits=8, K=97, blocks=200),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the ranges above: region to biobank panels, every form and option, few to many traits."""
    what = rng.choice(["int8", "int8", "int8", "sketch", "sketch", "fp64", "annot", "bed", "h2", "h2", "rg", "h2p"])
    if what in ("int8", "sketch", "fp64", "annot", "bed"):
        n = _log(rng, 1500, 60000)
        top = {"int8": 3.5e9, "sketch": 3e9, "fp64": 4e7, "annot": 1e9, "bed": 1e9}[what]
        per_cm = _log(rng, 140, 1300 if what != "fp64" else 500)
        m = _log(rng, 700, max(1500, min(100000, int(top / n))))
        c = dict(kind="bed" if what == "bed" else "l2", n=n, m=m, chroms=rng.choice([1, 1, 2, 5]), per_cm=per_cm,
                 form={"annot": "int8", "bed": "int8"}.get(what, what), masked=rng.random() < 0.6)
        if what == "sketch":
            c["d"] = min(_log(rng, 50, 5000), n // 4)
            c["maf_aware"] = rng.random() < 0.3
        if what == "annot":
            c["K"] = rng.choice([2, 10, 53, 97])
            c["on_device"] = rng.random() < 0.5
            c["form"] = rng.choice(["int8", "int8", "sketch"])
            if c["form"] == "sketch":
                c["d"] = min(1000, n // 4)
        if what in ("int8", "annot") and rng.random() < 0.35:
            c["keep"] = max(3, int(n * rng.uniform(0.3, 0.99)))
        if what in ("int8", "fp64") and rng.random() < 0.35:
            c["extract"] = True
        if rng.random() < 0.3:
            c["window"] = rng.choice(["kb", "snp"])
        if what != "bed" and rng.random() < 0.2:
            c["pq_exp"] = 1.0
        return c
    m = _log(rng, 5000, 250000)
    if what == "h2":
        c = dict(kind="h2", m=m, traits=_log(rng, 1, 600), blocks=200, lambda_gc=rng.random() < 0.7)
        if rng.random() < 0.4:  # a program with its arrays on the host, through h2_batch
            c.update(traits=_log(rng, 1, 20), host=True)
            if rng.random() < 0.5:
                c["two_step"] = 30.0
            if rng.random() < 0.5:
                c["n_per_snp"] = True
        return c
    if what == "rg":
        return dict(kind="rg", m=m, traits=_log(rng, 1, 150), blocks=200)
    return dict(kind="h2p", m=m, traits=_log(rng, 1, 6), K=rng.choice([2, 25, 53, 97]), blocks=200)


# ---- inputs (made from the seed alone) ----------------------------------------

def _rng(seed, salt):
    return np.random.default_rng([int(seed), salt])


def _gen(seed, salt):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed) * 1009 + salt)
    return g


def _positions(case, seed):
    """(chr, cM, bp) of the records: exponential gaps, about per_cm records a cM."""
    m, nc = case["m"], case["chroms"]
    cut = [m * c // nc for c in range(nc + 1)]
    gaps = _rng(seed, 1).exponential(1.0 / case["per_cm"], m)
    chr_, cm = np.zeros(m, np.uint8), np.zeros(m)
    for c in range(nc):
        s = slice(cut[c], cut[c + 1])
        chr_[s] = c + 1
        cm[s] = np.cumsum(gaps[s])
    return chr_, cm, (1 + np.floor(cm * 1e6)).astype(np.uint32)


def _rows(case, seed):
    """Panel rows of the records: every row, or with extract two of three (odd gaps)."""
    if not case.get("extract"):
        return np.arange(case["m"], dtype=np.int64), case["m"]
    rows = np.cumsum(_rng(seed, 2).integers(1, 3, case["m"])) - 1
    return rows.astype(np.int64), int(rows[-1]) + 3


def _kept_iids(case, seed):
    if not case.get("keep"):
        return None
    return np.sort(_rng(seed, 3).permutation(case["n"])[:case["keep"]]).astype(np.int64)


def _bed(case, seed):
    """The panel's BED body, (rows, ceil(n / 4)) uint8, on the GPU."""
    n, total = case["n"], _rows(case, seed)[1]
    g = _gen(seed, 4)
    dev = torch.device("cuda")
    p = 0.02 + 0.96 * torch.rand(total, generator=g, device=dev)
    table = (torch.rand(FOUNDERS, total, generator=g, device=dev) < p).to(torch.uint8)
    nseg = total // SEG + 2
    founder = torch.randint(0, FOUNDERS, (2 * n, nseg), generator=g, device=dev, dtype=torch.int16)
    phase = torch.randint(0, SEG, (2 * n,), generator=g, device=dev, dtype=torch.int32)
    bpr = (n + 3) // 4
    out = torch.empty((total, bpr), dtype=torch.uint8, device=dev)
    block = max(1, min(total, (1 << 25) // n))
    for b0 in range(0, total, block):
        b1 = min(total, b0 + block)
        # a haplotype changes founder once every SEG records, at its own phase
        code = torch.zeros((b1 - b0, 4 * bpr), dtype=torch.uint8, device=dev)
        for s in range(b0 // SEG, (b1 - 1) // SEG + 1):
            r0, r1 = max(b0, s * SEG), min(b1, (s + 1) * SEG)
            first, second = founder[:, s].long(), founder[:, s + 1].long()
            j = torch.arange(r0 - s * SEG, r1 - s * SEG, device=dev, dtype=torch.int32)
            t = table[:, r0:r1].t()
            a = torch.where(j[:, None] < phase[None, :], t[:, first], t[:, second])
            a = a[:, :n] + a[:, n:]
            code[r0 - b0:r1 - b0, :n] = 3 - a - a // 2   # genotype 0, 1, 2 -> code 3, 2, 0
        lost = torch.rand((b1 - b0, n), generator=g, device=dev) < 0.008
        code[:, :n][lost] = 1
        c4 = code.view(b1 - b0, bpr, 4)
        out[b0:b1] = c4[:, :, 0] | (c4[:, :, 1] << 2) | (c4[:, :, 2] << 4) | (c4[:, :, 3] << 6)
    return out


def _annotations(case, seed):
    """(K, m) float64 on the GPU: all ones, binary runs of 20 records, clipped normals."""
    K, m = case["K"], case["m"]
    g = _gen(seed, 5)
    dev = torch.device("cuda")
    a = torch.ones((K, m), dtype=torch.float64, device=dev)
    nb = max(0, (K - 1) * 5 // 6)
    if nb:
        dens = 0.01 + 0.19 * torch.rand((nb, 1), generator=g, device=dev)
        runs = (torch.rand((nb, m // 20 + 1), generator=g, device=dev) < dens).double()
        a[1:1 + nb] = runs.repeat_interleave(20, dim=1)[:, :m]
    if K - 1 - nb:
        x = torch.randn((K - 1 - nb, m), generator=g, device=dev, dtype=torch.float64)
        a[1 + nb:] = x.clamp(-3.0, 3.0)
    return a


M_SNPS = 1.2e6   # SNPs behind the LD scores of the regressions


def _ld_scores(case, seed):
    """(m,) LD scores, 1 to a few hundred."""
    m = case["m"]
    g = _gen(seed, 6)
    u = torch.rand(m, generator=g, device="cuda", dtype=torch.float64)
    v = torch.rand(m, generator=g, device="cuda", dtype=torch.float64)
    return 1.0 - 20.0 * torch.log(u + 1e-12) * (0.2 + v)


def _traits(case, seed, scores, salt):
    """Per trait h2 and N, and z-scores of a polygenic trait on the LD scores."""
    T, m = case["traits"], case["m"]
    g = _gen(seed, salt)
    f = dict(generator=g, device="cuda", dtype=torch.float64)
    h2 = 0.1 + 0.4 * torch.rand(T, **f)
    n = torch.exp(math.log(3e4) + math.log(15.0) * torch.rand(T, **f))
    b = torch.randn((T, m), **f)
    z = torch.sqrt(n[:, None] * h2[:, None] * scores[None, :] / M_SNPS) * b + torch.randn((T, m), **f)
    return z, n, h2, b


def _h2_inputs(case, seed):
    ld = _ld_scores(case, seed)
    z, n, _, _ = _traits(case, seed, ld, 7)
    n_snp = None
    if case.get("n_per_snp"):
        g = _gen(seed, 8)
        n_snp = n[:, None] * (0.8 + 0.2 * torch.rand(z.shape, generator=g, device="cuda", dtype=torch.float64))
    return dict(chi2=z * z, n=n, n_snp=n_snp, ld=ld, w=0.8 * ld + 0.5)


def _rg_inputs(case, seed):
    ld = _ld_scores(case, seed)
    z1, n1, _, b1 = _traits(case, seed, ld, 9)
    g = _gen(seed, 10)
    f = dict(generator=g, device="cuda", dtype=torch.float64)
    T, m = case["traits"], case["m"]
    rg = 1.6 * torch.rand(T, **f) - 0.8
    h2, n2 = 0.1 + 0.4 * torch.rand(T, **f), torch.exp(math.log(3e4) + math.log(15.0) * torch.rand(T, **f))
    b2 = rg[:, None] * b1 + torch.sqrt(1.0 - rg * rg)[:, None] * torch.randn((T, m), **f)
    z2 = torch.sqrt(n2[:, None] * h2[:, None] * ld[None, :] / M_SNPS) * b2 + torch.randn((T, m), **f)
    return dict(z1=z1, z2=z2, n1=n1, n2=n2, ld=ld, w=0.8 * ld + 0.5)


def _h2p_inputs(case, seed):
    K, m = case["K"], case["m"]
    base = _ld_scores(case, seed)
    g = _gen(seed, 11)
    f = dict(generator=g, device="cuda", dtype=torch.float64)
    l2 = torch.empty((K, m), dtype=torch.float64, device="cuda")
    l2[0] = base
    if K > 1:
        share = 0.02 + 0.3 * torch.rand((K - 1, 1), **f)
        l2[1:] = base * share * (0.1 - torch.log(torch.rand((K - 1, m), **f) + 1e-12))
    z, n, _, _ = _traits(case, seed, base, 12)
    chi2 = z * z
    m_vec = np.concatenate([[M_SNPS], _rng(seed, 13).uniform(0.02, 0.3, K - 1) * M_SNPS])
    return dict(chi2=chi2, n=n, l2=l2, w=base, m_vec=m_vec, cmax=np.maximum(0.001 * n.cpu().numpy(), 80.0))


# ---- the calls -----------------------------------------------------------------

def _context():
    if "ctx" not in _kept:
        from ldsc_b200.api import Context
        _kept["ctx"] = Context(0)
    return _kept["ctx"]


def _server():
    if "srv" not in _kept:
        from ldsc_b200.serve import Server
        _kept["srv"] = Server(0, n_slots=1)
    return _kept["srv"]


def _window(case):
    from ldsc_b200.api import WindowMode
    w = case.get("window", "cm")
    if w == "kb":
        return WindowMode.Kb(1000.0)
    if w == "snp":
        return WindowMode.Snp(case["per_cm"])
    return WindowMode.Cm(1.0)


def _host(t):
    return t.cpu().numpy()


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("l2", "bed"):
        from ldsc_b200.plink import BimTable
        ctx = _context()
        chr_, cm, bp = _positions(case, seed)
        rows, total = _rows(case, seed)
        s = dict(kind=kind, ctx=ctx, case=case, mode=_window(case), keep=_kept_iids(case, seed),
                 snps=BimTable(chr_, [f"rs{i}" for i in range(case["m"])], cm, bp, rows))
        body = _bed(case, seed)
        if kind == "bed":
            bpr = (case["n"] + 3) // 4
            image = torch.empty(3 + total * bpr, dtype=torch.uint8, pin_memory=True)
            image[:3] = torch.tensor([0x6C, 0x1B, 0x01], dtype=torch.uint8)
            image[3:] = body.view(-1).cpu()
            s["image"], s["buffer"] = image.numpy(), image
        else:
            s["panel"] = ctx.upload(_host(body), case["n"])
        if case.get("K"):
            a = _annotations(case, seed)
            if case.get("on_device"):
                s["annot"] = a
                s["l2"] = torch.empty((case["K"], case["m"]), dtype=torch.float64, device="cuda")
                s["maf"] = torch.empty(case["m"], dtype=torch.float64, device="cuda")
            else:
                s["annot"] = np.asfortranarray(_host(a).T)
        return s
    if kind == "h2":
        x = _h2_inputs(case, seed)
        if case.get("host"):
            return dict(kind=kind, case=case, ctx=_context(), **{k: None if v is None else _host(v) for k, v in x.items()})
        return dict(kind=kind, case=case, srv=_server(), **x)
    if kind == "rg":
        return dict(kind=kind, case=case, srv=_server(), **_rg_inputs(case, seed))
    return dict(kind=kind, case=case, srv=_server(), **_h2p_inputs(case, seed))


def run(s):
    case, kind = s["case"], s["kind"]
    if kind == "l2":
        from ldsc_b200.api import run_l2
        dev = bool(case.get("on_device"))
        annot = s.get("annot")
        l2, maf, _ = run_l2(
            s["ctx"], s["snps"], s["panel"], s["mode"], 200, annot=None if dev else annot, iid_indices=s["keep"],
            pq_exp=case.get("pq_exp"), yes_really=True, sketch=case.get("d"),
            sketch_maf_aware=bool(case.get("maf_aware")), snp_level_masking=case["masked"],
            precision="int8" if case["form"] == "int8" else "fp64",
            annot_device=(annot.data_ptr(), case["m"], case["K"]) if dev else None,
            out_device=(s["l2"], s["maf"]) if dev else None)
        return {"l2": l2, "maf": maf}
    if kind == "bed":
        from ldsc_b200.api import l2_from_bed_bytes
        l2, maf, _ = l2_from_bed_bytes(s["ctx"], s["image"], case["n"], s["snps"], s["mode"], 200, precision="int8",
                                       snp_level_masking=case["masked"])
        return {"l2": l2, "maf": maf}
    if kind == "h2" and case.get("host"):
        from ldsc_b200.api import h2_batch
        out = h2_batch(s["ctx"], s["chi2"], s["n"] if s["n_snp"] is None else s["n_snp"], s["ld"], s["w"], M_SNPS,
                       case["blocks"], lambda_gc=case["lambda_gc"], two_step=case.get("two_step"))
    elif kind == "h2":
        srv = s["srv"]
        out, _ = srv.wait(srv.submit_h2(s["chi2"], s["n"], s["ld"], s["w"], M_SNPS, case["blocks"],
                                        lambda_gc=case["lambda_gc"]))
    elif kind == "rg":
        srv = s["srv"]
        out, _ = srv.wait(srv.submit_rg(s["z1"], s["z2"], s["n1"], s["n2"], s["ld"], s["w"], M_SNPS, case["blocks"]))
    else:
        srv = s["srv"]
        fits, _ = srv.wait(srv.submit_h2_partitioned(s["chi2"], s["n"], s["l2"], s["w"], s["m_vec"], s["cmax"],
                                                     case["blocks"]))
        return {"est": np.stack([f.est for f in fits]), "cov": np.stack([f.cov for f in fits]),
                "delete_values": np.stack([f.delete_values for f in fits]),
                "h2_annot": np.stack([f.h2_annot for f in fits]),
                "totals": np.array([[f.h2_total, f.h2_total_se, f.intercept, f.intercept_se, f.n_mean, f.mean_chi2]
                                    for f in fits]),
                "n_obs": np.array([f.n_obs for f in fits])}
    return {name: np.ascontiguousarray(out[name]) for name in out.dtype.names}


# ---- what a pass cannot do without -----------------------------------------------

def work(case):
    kind = case["kind"]
    if kind in ("l2", "bed"):
        n = case.get("keep") or case["n"]
        left = _left_limits(case, *_positions(case, 0))
        pairs = float((np.arange(case["m"]) - left).sum())
        K = case.get("K", 1)
        nbytes = case["m"] * ((case["n"] + 3) // 4) + 8.0 * case["m"] * (2 + (2 * K if case.get("K") else K))
        flops = 2.0 * pairs * (case["d"] if case["form"] == "sketch" else n)
        if case.get("K"):
            flops += 4.0 * pairs * K
        return {"bytes": nbytes, "flops": flops}
    T, m = case["traits"], case["m"]
    if kind == "h2":
        return {"bytes": 8.0 * T * m * (2 if case.get("n_per_snp") else 1) + 16.0 * m, "flops": 40.0 * T * m}
    if kind == "rg":
        return {"bytes": 16.0 * T * m + 16.0 * m, "flops": 120.0 * T * m}
    P = case["K"] + 1
    return {"bytes": 8.0 * T * m + 8.0 * (case["K"] + 1) * m,
            "flops": 1.0 * T * (m * P * P + case["blocks"] * 2.0 * P ** 3 / 3.0)}


# ---- the values in 64 bits ---------------------------------------------------------

def _left_limits(case, chr_, cm, bp):
    m = case["m"]
    left = np.zeros(m, np.int64)
    edges = np.flatnonzero(np.r_[True, chr_[1:] != chr_[:-1], True])
    for s, e in zip(edges[:-1], edges[1:]):
        i = np.arange(e - s)
        w = case.get("window", "cm")
        if w == "snp":
            lo = np.maximum(i - case["per_cm"], 0)
        else:
            x, size = (cm[s:e], 1.0) if w == "cm" else (bp[s:e].astype(np.float64) / 1000.0, 1000.0)
            lo = np.searchsorted(x, x - size, side="left")
            for _ in range(3):   # the window is on the rounded difference
                back = (lo > 0) & (x - x[np.maximum(lo - 1, 0)] <= size)
                lo = lo - back
                lo = lo + (x - x[lo] > size)
        if case["masked"]:
            left[s:e] = s + lo
        else:
            for c0 in range(0, e - s, 200):
                dist = c0 - lo[c0]
                left[s + c0:min(e, s + c0 + 200)] = s + c0 - min(c0, -(-dist // 200) * 200)
    return left


def _standardised(code):
    """2-bit codes (records, individuals) -> (standardised f64 rows, maf, kurtosis term)."""
    g = torch.tensor([2.0, 0.0, 1.0, 0.0], dtype=torch.float64, device=code.device)[code.long()]
    here = (code != 1).double()
    n = here.sum(1)
    mean = torch.where(n > 0, g.sum(1) / n.clamp(min=1.0), 0.0 * n)
    x = (g - mean[:, None]) * here
    css = (x * x).sum(1)
    kappa = torch.where(css > 0, (x ** 4).sum(1) / (css * css).clamp(min=1e-300), 0.0 * css)
    inv = torch.where(css > 0, torch.rsqrt((css / code.shape[1]).clamp(min=1e-300)), 0.0 * css)
    freq = (mean / 2.0).clamp(0.0, 1.0)
    return x * inv[:, None], torch.minimum(freq, 1.0 - freq), kappa


def _seed42_stream(n, d):
    """Bucket and sign per individual: the WyRand generator seeded with 42, buckets by
    multiply-shift with rejection, then one coin per individual."""
    full = (1 << 64) - 1
    state = 42

    def step():
        nonlocal state
        state = (state + 0x2D358DCCAA6C78A5) & full
        t = state * (state ^ 0x8BB84B93962EACC9)
        return (t & full) ^ (t >> 64)

    bucket = np.zeros(n, np.int64)
    for i in range(n):
        p = (step() & 0xFFFFFFFF) * d
        if (p & 0xFFFFFFFF) < d:
            least = ((1 << 32) - d) % d
            while (p & 0xFFFFFFFF) < least:
                p = (step() & 0xFFFFFFFF) * d
        bucket[i] = p >> 32
    sign = np.array([1.0 if (step() & 0xFF) % 2 == 0 else -1.0 for _ in range(n)])
    return torch.from_numpy(bucket).cuda(), torch.from_numpy(sign).cuda()


def _exact_l2(case, seed):
    dev = torch.device("cuda")
    m = case["m"]
    body = _bed(case, seed)
    body = body[torch.from_numpy(_rows(case, seed)[0]).to(dev)]
    keep = _kept_iids(case, seed)
    keep = None if keep is None else torch.from_numpy(keep).to(dev)
    n = case["n"] if keep is None else len(keep)
    sketch = case["form"] == "sketch"
    bucket, sign = _seed42_stream(n, case["d"]) if sketch else (None, None)
    left = _left_limits(case, *_positions(case, seed))
    step = max(64, min(1024, int(1.2e8 / n)))
    width = case["d"] if sketch else n
    maf, kappa = torch.zeros(m, dtype=torch.float64, device=dev), torch.zeros(m, dtype=torch.float64, device=dev)

    def rows(b0, b1):
        b = body[b0:b1]
        code = torch.stack([(b >> s) & 3 for s in (0, 2, 4, 6)], dim=2).reshape(b1 - b0, -1)[:, :case["n"]]
        code = code if keep is None else code[:, keep]
        x, maf[b0:b1], kappa[b0:b1] = _standardised(code)
        if sketch:
            x = torch.zeros((b1 - b0, width), dtype=torch.float64, device=dev).index_add_(1, bucket, x * sign)
            norm = (x * x).sum(1)
            x = torch.where(norm[:, None] > 0, x * torch.sqrt(n / norm.clamp(min=1e-300))[:, None], x)
        return x

    denom = n - 2.0 if n > 2 else float(n)
    L = torch.from_numpy(left).to(dev)
    idx = torch.arange(m, device=dev)
    blocks, tiles = {}, []
    maf_all_first = case.get("pq_exp") is not None
    if maf_all_first:
        for b0 in range(0, m, step):
            rows(b0, min(m, b0 + step))
    a = torch.ones((1, m), dtype=torch.float64, device=dev) if not case.get("K") else _annotations(case, seed)
    if maf_all_first:
        a = a * (maf * (1.0 - maf)) ** case["pq_exp"]
    l2 = a.clone()
    for b0 in range(0, m, step):
        b1 = min(m, b0 + step)
        blocks[b0] = rows(b0, b1)
        first = int(left[b0:b1].min())
        for k0 in [k for k in blocks if k + step <= first]:
            del blocks[k0]
        for k0 in sorted(blocks):
            k1 = min(m, k0 + step)
            r = blocks[k0] @ blocks[b0].T
            t = (r / n) ** 2
            if sketch:
                d = float(case["d"])
                kap = kappa[k0:k1, None] + kappa[None, b0:b1] if case.get("maf_aware") else 0.0
                dm3 = d - 3.0 - 2.0 * kap
                disc = dm3 * dm3 + 8.0 * (d * t - 1.0)
                t = torch.where(disc >= 0, (-dm3 + torch.sqrt(disc.clamp(min=0.0))) * 0.25, 0.0 * t)
            t = t * (1.0 + 1.0 / denom) - 1.0 / denom
            inside = (idx[k0:k1, None] < idx[None, b0:b1]) & (idx[k0:k1, None] >= L[None, b0:b1])
            t = torch.where(inside, t, 0.0 * t)
            l2[:, b0:b1] += a[:, k0:k1] @ t
            l2[:, k0:k1] += a[:, b0:b1] @ t.T
    if case.get("on_device"):
        return {"l2": l2, "maf": maf}
    return {"l2": l2.T.contiguous(), "maf": maf}


def _cuts(m, nb):
    return [int(math.floor(b * m / nb)) for b in range(nb)] + [m]


def _block_sums(v, cuts):
    c = torch.tensor(cuts, device=v.device)
    at = c[:-1, None] + torch.arange(int((c[1:] - c[:-1]).max()), device=v.device)
    return torch.where(at < c[1:, None], v[at.clamp(max=len(v) - 1)], 0.0 * v[0]).sum(1)


class _Fit:
    """One weighted regression of y on [x, 1]: two re-weightings, then the block jackknife."""

    def __init__(self, y, nx, ld, weight, nb, m_snps, int0, fixed=None, keep=None, cuts=None):
        self.mean_y, self.nbar = y.mean(), nx.mean()
        self.slope = m_snps * (self.mean_y - int0) / (ld * nx).mean()
        self.intercept = int0
        x = nx * ld / self.nbar
        inside = torch.ones_like(y) if keep is None else keep.double()
        self.first = None
        for it in range(3):
            w = weight(self.slope, self.intercept, it) * inside
            S = [(w * x * x).sum(), (w * x).sum(), w.sum(), (w * x * y).sum(), (w * y).sum()]
            if it == 0:
                self.first = (S[1], S[0])
            if it < 2:
                e0, e1 = self.solve(S, fixed)
                self.slope, self.intercept = m_snps * e0 / self.nbar, e1
        cuts = cuts or _cuts(len(y), nb)
        B = [_block_sums(v, cuts) for v in (w * x * x, w * x, w, w * x * y, w * y)]
        S = [v.sum() for v in B]
        self.est = torch.stack([torch.as_tensor(v, dtype=torch.float64, device=y.device) for v in self.solve(S, fixed)])
        d0, d1 = self.solve([s - b for s, b in zip(S, B)], fixed)
        self.delete = torch.stack([d0, d1 if torch.is_tensor(d1) and d1.dim() else torch.full_like(d0, float(d1))])
        self.cov = _jack(self.est, self.delete)

    @staticmethod
    def solve(S, fixed):
        a, b, c, d, e = S
        if fixed is not None:
            return (d - fixed * b) / a, fixed
        det = a * c - b * b
        return (c * d - b * e) / det, (a * e - b * d) / det


def _jack(est, delete):
    """Jackknife covariance of est (P) from delete values (P, nb)."""
    nb = delete.shape[1]
    pseudo = nb * est[:, None] - (nb - 1.0) * delete
    c = pseudo - pseudo.mean(1, keepdim=True)
    return c @ c.T / (nb * (nb - 1.0))


def _h2_weight(n, ld, w_ld):
    def weight(slope, intercept, it):
        t = intercept + torch.clamp(slope, 0.0, 1.0) * n * ld.clamp(min=1.0) / M_SNPS
        return 1.0 / (2.0 * t * t * w_ld.clamp(min=1.0))
    return weight


def _exact_h2(case, seed):
    x = _h2_inputs(case, seed)
    names = ("h2", "h2_se", "intercept", "intercept_se", "mean_chi2", "lambda_gc", "ratio", "ratio_se", "coef", "coef_se")
    out = {k: [] for k in names}
    nb, ld = case["blocks"], x["ld"]
    for t in range(case["traits"]):
        y = x["chi2"][t]
        n = x["n"][t] * torch.ones_like(y) if x["n_snp"] is None else x["n_snp"][t]
        plain = _h2_weight(n, ld, x["w"])
        if case.get("two_step"):
            kept = y < case["two_step"]
            at = torch.nonzero(kept)[:, 0]
            nk = len(at)
            cuts = [0] + [int(at[b * nk // nb]) for b in range(1, nb)] + [len(y)]

            def on_x(slope, intercept, it, n=n, nbar=n.mean()):
                return plain(slope, intercept, it) if it == 0 else _h2_weight(n, n * ld / nbar, x["w"])(slope, intercept, it)

            f1 = _Fit(y, n, ld, on_x, nb, M_SNPS, 1.0, keep=kept, cuts=cuts)
            f2 = _Fit(y, n, ld, plain, nb, M_SNPS, 1.0, fixed=f1.est[1], cuts=cuts)
            c = f2.first[0] / f2.first[1]
            est = torch.stack([f2.est[0], f1.est[1]])
            delete = torch.stack([f2.delete[0] - c * (f1.delete[1] - f1.est[1]), f1.delete[1]])
            cov, f = _jack(est, delete), f2
        else:
            f = _Fit(y, n, ld, plain, nb, M_SNPS, 1.0)
            est, cov = f.est, f.cov
        se, k = torch.sqrt(torch.diagonal(cov)), M_SNPS / f.nbar
        q = torch.sort(y).values
        med = (q[(len(y) - 1) // 2] + q[len(y) // 2]) / 2.0
        ok = bool(f.mean_y > 1.0)
        nan = torch.full_like(se[0], math.nan)
        for name, v in zip(names, (k * est[0], k * se[0], est[1], se[1], f.mean_y, med / 0.4549 if case["lambda_gc"] else nan,
                                   (est[1] - 1.0) / (f.mean_y - 1.0) if ok else nan, se[1] / (f.mean_y - 1.0) if ok else nan,
                                   est[0] / f.nbar, se[0] / f.nbar)):
            out[name].append(v)
    return {k: torch.stack(v) for k, v in out.items()}


def _exact_rg(case, seed):
    x = _rg_inputs(case, seed)
    names = ("rg", "rg_se", "z", "p", "gencov", "gencov_se", "gencov_intercept", "gencov_intercept_se", "h2_1",
             "h2_1_se", "h2_2", "h2_2_se", "mean_z1z2")
    out = {k: [] for k in names}
    nb, ld = case["blocks"], x["ld"]
    for t in range(case["traits"]):
        z1, z2 = x["z1"][t], x["z2"][t]
        fits = []
        for z, n in ((z1, x["n1"][t]), (z2, x["n2"][t])):
            nn = n * torch.ones_like(z)
            fits.append(_Fit(z * z, nn, ld, _h2_weight(nn, ld, x["w"]), nb, M_SNPS, 1.0))
        f1, f2 = fits
        h1, h2 = M_SNPS * f1.est[0] / f1.nbar, M_SNPS * f2.est[0] / f2.nbar
        n1, n2 = x["n1"][t], x["n2"][t]
        root = torch.sqrt(n1 * n2)

        def weight(slope, intercept, it):
            l1 = ld.clamp(min=1.0)
            a = n1 * h1.clamp(0.0, 1.0) * l1 / M_SNPS + f1.est[1]
            b = n2 * h2.clamp(0.0, 1.0) * l1 / M_SNPS + f2.est[1]
            c = root * slope * l1 / M_SNPS + intercept
            return 1.0 / ((a * b + c * c) * x["w"].clamp(min=1.0))

        fg = _Fit(z1 * z2, root * torch.ones_like(z1), ld, weight, nb, M_SNPS, 0.0)
        tot, se = [], []
        for f in (f1, f2, fg):
            tot.append(M_SNPS * f.est[0] / f.nbar)
            se.append(M_SNPS * torch.sqrt(f.cov[0, 0]) / f.nbar)
        rg = tot[2] / torch.sqrt(tot[0] * tot[1])
        d = [M_SNPS * f.delete[0] / f.nbar for f in (f1, f2, fg)]
        rg_se = torch.sqrt(_jack(rg[None], (d[2] / torch.sqrt(d[0] * d[1]))[None])[0, 0])
        zz = rg / rg_se
        for name, v in zip(names, (rg, rg_se, zz, torch.erfc(zz.abs() / math.sqrt(2.0)), tot[2], se[2], fg.est[1],
                                   torch.sqrt(fg.cov[1, 1]), tot[0], se[0], tot[1], se[1], fg.mean_y)):
            out[name].append(v)
    return {k: torch.stack(v) for k, v in out.items()}


def _exact_h2p(case, seed):
    x = _h2p_inputs(case, seed)
    nb, K = case["blocks"], case["K"]
    out = {k: [] for k in ("est", "cov", "delete_values", "h2_annot", "totals", "n_obs")}
    m_vec = torch.from_numpy(x["m_vec"]).cuda()
    m_tot = m_vec.sum()
    xt_all = x["l2"].sum(0)
    for t in range(case["traits"]):
        kept = x["chi2"][t] < float(x["cmax"][t])
        y, l2, xt, w_ld = x["chi2"][t][kept], x["l2"][:, kept], xt_all[kept], x["w"][kept]
        n = float(x["n"][t])
        hsq = m_tot * (y.mean() - 1.0) / (xt * n).mean()
        s = 1.0 + hsq.clamp(0.0, 1.0) * n / m_tot * xt.clamp(min=1.0)
        w = 1.0 / (2.0 * s * s) / w_ld.clamp(min=1.0)
        z = torch.cat([l2, torch.ones_like(y)[None], y[None]])   # N / nbar = 1
        cuts = _cuts(len(y), nb)
        G = torch.stack([(z[:, cuts[b]:cuts[b + 1]] * w[cuts[b]:cuts[b + 1]]) @ z[:, cuts[b]:cuts[b + 1]].T
                         for b in range(nb)])
        tot = G.sum(0)
        A = torch.cat([tot[None] - G, tot[None]])
        sol = torch.linalg.solve(A[:, :-1, :-1], A[:, :-1, -1])
        est, dv = sol[-1], sol[:-1]
        cov = _jack(est, dv.T.contiguous())
        h2 = est[:K] / n * m_vec
        var = (m_vec[:, None] * m_vec[None] * cov[:K, :K]).sum() / (n * n)
        for name, v in zip(out, (est, cov, dv, h2, torch.stack([h2.sum(), torch.sqrt(var.clamp(min=0.0)), est[K],
                                                                torch.sqrt(cov[K, K]), torch.full_like(var, n), y.mean()]),
                                 torch.tensor(len(y)))):
            out[name].append(v)
    return {k: torch.stack(v) for k, v in out.items()}


def exact(case, seed):
    if case["kind"] in ("l2", "bed"):
        return _exact_l2(case, seed)
    return {"h2": _exact_h2, "rg": _exact_rg, "h2p": _exact_h2p}[case["kind"]](case, seed)
