"""Timed cases of the polygenic-score framework: scoring, refitting, .pgen decode, projection.

Every case goes through the package's public entry points.  Genotypes follow
Hardy-Weinberg with allele frequencies 0.01-0.5 and a missing rate of 0.5-2 %,
weights are normal with sigma 0.01, a tenth of the cells has its alleles
flipped: the distributions of the repository's named workloads.  Inputs are
made with torch on the GPU from the seed alone.
"""
import math

import numpy as np
import torch

from gnomon_b200 import synth
from gnomon_b200.autograd import polygenic_score, prep_from_dense
from gnomon_b200.device import DevicePlan, row_pitch
from gnomon_b200.pgen import PgenFile
from gnomon_b200.pipeline import PipelineContext, run as pipeline_run
from gnomon_b200.prepare import PreparationResult
from gnomon_b200.project import Projector, hwe_coefficients

DEVICE = "cuda"
CHUNK = 1 << 27          # genotypes handled at once while making inputs
P_LO, P_HI, SIGMA, FLIP = 0.01, 0.5, 0.01, 0.10


# ---- cases ------------------------------------------------------------------------


def listed():
    return [
        # one score on a clinic-sized cohort: a single call is all latency and launches
        dict(name="score_clinic_k1", kind="score", people=2_000, variants=50_000, scores=1,
             missing=0.01, cover=1.0, keep=1.0),
        # a handful of scores on a small ragged cohort (tensor engine, launch bound)
        dict(name="score_small_k12", kind="score", people=1_503, variants=30_011, scores=12,
             missing=0.01, cover=1.0, keep=1.0),
        # one genome-wide score on a large cohort: the repository's bandwidth workload
        dict(name="score_cohort_k1", kind="score", people=50_000, variants=1_000_000, scores=1,
             missing=0.005, cover=1.0, keep=1.0),
        # a panel of four scores of uneven sizes, with a keep list, ragged sizes
        dict(name="score_panel_k4", kind="score", people=30_011, variants=150_007, scores=4,
             missing=0.01, cover=0.2, keep=0.9),
        # the forward half of the repository's differentiation workload
        dict(name="score_k16", kind="score", people=20_000, variants=200_000, scores=16,
             missing=0.01, cover=1.0, keep=1.0),
        # a resident block of the biobank workload: 64 uneven scores
        dict(name="score_biobank_k64", kind="score", people=200_000, variants=60_000, scores=64,
             missing=0.02, cover=0.02, keep=1.0),
        # a block of the catalogue workload: 512 uneven scores in one pass
        dict(name="score_catalog_k512", kind="score", people=100_000, variants=40_000, scores=512,
             missing=0.01, cover=0.02, keep=1.0),
        # the backward half of the differentiation workload: dW and d(correction)
        dict(name="backward_k16", kind="backward", people=20_000, variants=200_000, scores=16,
             missing=0.01, keep=1.0),
        # one step of refitting three scores on a ragged cohort through autograd
        dict(name="refit_step_k3", kind="refit", people=4_001, variants=20_011, scores=3,
             missing=0.01),
        # a resident PLINK 2 file with linkage, decoded into rows on the device
        dict(name="pgen_decode", kind="pgen", people=50_000, variants=256, repeats=64,
             missing=0.01),
        # PCA projection of a cohort from host memory, two blocks of variants
        dict(name="project_k20", kind="project", people=50_000, variants=4_096, blocks=2, axes=20,
             missing=0.01),
        # the whole scoring call on a .bed in host memory that holds more rows than needed
        dict(name="run_bed_k3", kind="run", people=20_003, variants=60_000, scores=3,
             missing=0.01, cover=0.5),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """A case of the ranges that listed() stands for; sizes log-uniform, mostly odd."""
    u = rng.random()
    missing = rng.choice([0.005, 0.01, 0.02])
    if u < 0.60:
        k = rng.choice([1, 1, 2, 3, 5, 7, _log(rng, 8, 64), _log(rng, 8, 64), _log(rng, 65, 512)])
        people, variants = _log(rng, 500, 200_000), _log(rng, 2_000, 1_000_000)
        # no dearer than the listed cases of the same number of scores
        most = (5e10 if k == 1 else 4e10 / k if k < 8 else 4e10 / ((k + 15) // 16) if k <= 64
                else 8e9 / ((k + 127) // 128))
        variants = max(1_000, int(min(variants, most / people, 2e7 / k)))
        return dict(kind="score", people=people, variants=variants, scores=k, missing=missing,
                    cover=rng.choice([1.0, 0.2, 0.02]), keep=rng.choice([1.0, 0.9, 0.5]))
    if u < 0.75:
        k = rng.choice([1, 3, 8, 16, 16, 24])
        people = _log(rng, 500, 50_000)
        variants = int(min(_log(rng, 2_000, 200_000), 4e9 / people / ((k + 15) // 16)))
        return dict(kind="backward", people=people, variants=variants, scores=k, missing=missing,
                    keep=rng.choice([1.0, 0.8]))
    if u < 0.83:
        return dict(kind="refit", people=_log(rng, 500, 8_000), variants=_log(rng, 2_000, 20_000),
                    scores=rng.choice([1, 2, 3, 5]), missing=missing)
    if u < 0.90:
        return dict(kind="pgen", people=_log(rng, 2_000, 50_000), variants=rng.choice([128, 256]),
                    repeats=rng.choice([16, 32, 64]), missing=missing)
    if u < 0.95:
        return dict(kind="project", people=_log(rng, 2_000, 50_000),
                    variants=_log(rng, 500, 4_096), blocks=rng.choice([1, 2]),
                    axes=rng.choice([4, 10, 20]), missing=missing)
    return dict(kind="run", people=_log(rng, 2_000, 20_000), variants=_log(rng, 5_000, 60_000),
                scores=rng.choice([1, 3, 12]), missing=missing, cover=rng.choice([1.0, 0.5]))


# ---- inputs -----------------------------------------------------------------------


def _rows(gen, people, variants, missing, pitch):
    """Packed SNP-major rows [variants * pitch] (person i at bits 2 * (i % 4)) on the GPU."""
    bpv = (people + 3) // 4
    rows = torch.zeros((variants, pitch), dtype=torch.uint8, device=DEVICE)
    freq = P_LO + (P_HI - P_LO) * torch.rand(variants, 1, generator=gen, device=DEVICE)
    shift = torch.tensor([1, 4, 16, 64], dtype=torch.uint8, device=DEVICE)
    step = max(1, min(variants, CHUNK // (4 * bpv)))
    for v in range(0, variants, step):
        p = freq[v:v + step]
        n = len(p)
        u = torch.rand(n, 4 * bpv, generator=gen, device=DEVICE)
        u[:, people:] = missing                       # past the last person: code 00
        ref = missing + (1 - missing) * (1 - p) ** 2
        het = missing + (1 - missing) * (1 - p * p)
        codes = (u >= ref).to(torch.uint8).mul_(2).add_((u >= het).to(torch.uint8))
        codes += (u < missing)                        # 01: missing
        rows[v:v + n, :bpv] = (codes.view(n, bpv, 4) * shift).sum(-1, dtype=torch.uint8)
    return rows.view(-1)


def _cells(rng, variants, scores, cover):
    """(weights, flipped, member), each [variants][scores]: score k covers a share of the
    variants that rises from `cover` to all of them."""
    share = np.linspace(cover, 1.0, scores) if scores > 1 else np.ones(1)
    shape = (variants, scores)
    w = rng.standard_normal(shape, dtype=np.float32) * np.float32(SIGMA)
    flipped = rng.random(shape, dtype=np.float32) < FLIP
    member = rng.random(shape, dtype=np.float32) < share.astype(np.float32)
    return w, flipped, member


def _share(case):
    return (1 + case.get("cover", 1.0)) / 2 if case["scores"] > 1 else 1.0


def _prep(w, flipped, member, people, keep=None, required=None):
    if keep is None and required is None and member.all():
        return prep_from_dense(w, flipped, member, people)
    V, K = w.shape
    rows, cols = np.nonzero(member)
    ww, ff = w[rows, cols], flipped[rows, cols]
    dosage = np.where(ff, -ww, ww).astype(np.float32)
    corr = np.where(ff, np.float32(2) * ww, np.float32(0)).astype(np.float32)
    offs = np.zeros(V + 1, np.uint64)
    np.cumsum(member.sum(axis=1), out=offs[1:])
    return PreparationResult(dosage, corr, cols.astype(np.uint32), offs,
                             ["S%03d" % k for k in range(K)], people,
                             required_bim_indices=required, output_idx_to_fam_idx=keep,
                             baseline=np.bincount(cols, weights=corr, minlength=K))


def _keep(rng, people, share):
    if share >= 1.0:
        return None
    return np.sort(rng.permutation(people)[:max(1, int(people * share))]).astype(np.uint32)


def _sources(case, seed):
    gen = torch.Generator(device=DEVICE)
    gen.manual_seed(seed)
    return gen, np.random.default_rng(seed)


def _inputs(case, seed):
    """What a case is made of before any plan or handle: a dict of arrays."""
    gen, rng = _sources(case, seed)
    P, V, kind = case["people"], case["variants"], case["kind"]
    if kind in ("score", "backward", "refit"):
        pitch = row_pitch((P + 3) // 4)
        d = dict(pitch=pitch, rows=_rows(gen, P, V, case["missing"], pitch))
        d["w"], d["flipped"], d["member"] = _cells(rng, V, case["scores"], case.get("cover", 1.0))
        d["keep"] = _keep(rng, P, case.get("keep", 1.0))
        n = P if d["keep"] is None else len(d["keep"])
        d["grad"] = torch.randn(n, case["scores"], generator=gen, device=DEVICE)
        return d
    if kind == "run":
        bpv = (P + 3) // 4
        d = dict(rows=_rows(gen, P, V, case["missing"], bpv).cpu().numpy())
        d["required"] = np.sort(rng.permutation(V)[:int(0.9 * V)]).astype(np.uint64)
        d["w"], d["flipped"], d["member"] = _cells(rng, len(d["required"]), case["scores"],
                                                   case["cover"])
        return d
    if kind == "project":
        bpv = (P + 3) // 4
        n = case["blocks"] * V
        rows = _rows(gen, P, n, case["missing"], bpv).view(n, bpv).cpu().numpy()
        freq = rng.uniform(P_LO, P_HI, n)
        coeffs = hwe_coefficients(freq, np.sqrt(2 * freq * (1 - freq)), swapped=rng.random(n) < 0.1)
        loadings = rng.standard_normal((n, case["axes"])).astype(np.float32) / np.float32(n) ** 0.5
        return dict(rows=rows, coeffs=coeffs, loadings=loadings)
    # .pgen: categories in runs of 17 variants that copy their predecessor but for 2 % of the
    # people (REF and ALT swapped every fifth variant), so most records are LD-compressed
    p = P_LO + (P_HI - P_LO) * torch.rand(V, 1, generator=gen, device=DEVICE)
    u = torch.rand(V, P, generator=gen, device=DEVICE)
    base = ((u >= (1 - p) ** 2).to(torch.uint8) + (u >= 1 - p * p).to(torch.uint8))
    base[torch.rand(V, P, generator=gen, device=DEVICE) < case["missing"]] = 3
    redraw = torch.rand(V, P, generator=gen, device=DEVICE) < 0.02
    swap = torch.tensor([2, 1, 0, 3], dtype=torch.uint8, device=DEVICE)
    cats = base.clone()
    for v in range(1, V):
        if v % 17:
            prev = swap[cats[v - 1].long()] if v % 5 == 0 else cats[v - 1]
            cats[v] = torch.where(redraw[v], base[v], prev)
    return dict(pgen=synth.encode_pgen(cats.cpu().numpy(), case["repeats"]))


def prepare(case, seed):
    d = _inputs(case, seed)
    kind, P = case["kind"], case["people"]
    state = dict(case=case)
    if kind in ("score", "backward"):
        prep = _prep(d["w"], d["flipped"], d["member"], P, d["keep"])
        state |= dict(plan=DevicePlan(prep), rows=d["rows"], pitch=d["pitch"], grad=d["grad"])
    elif kind == "refit":
        state |= dict(rows=d["rows"], pitch=d["pitch"],
                      weights=torch.from_numpy(d["w"]).to(DEVICE).requires_grad_(True),
                      flipped=torch.from_numpy(d["flipped"]).to(DEVICE),
                      member=torch.from_numpy(d["member"]).to(DEVICE),
                      target=d["grad"].to(torch.float64))
    elif kind == "run":
        prep = _prep(d["w"], d["flipped"], d["member"], P, required=d["required"])
        state |= dict(context=PipelineContext(prep), rows=d["rows"])
    elif kind == "project":
        state |= d
    else:
        pg = PgenFile(d["pgen"])
        pitch = row_pitch(pg.bytes_per_variant)
        state |= dict(pgen=pg, pitch=pitch,
                      rows=torch.zeros(pg.variants * pitch, dtype=torch.uint8, device=DEVICE))
    return state


# ---- one pass ---------------------------------------------------------------------


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "score":
        sums, counts = state["plan"].score(state["rows"], state["pitch"])
        return {"sums": sums, "counts": counts}
    if kind == "backward":
        gw, gc = state["plan"].backward(state["rows"], state["pitch"], state["grad"],
                                        grad_corr=True)
        return {"weights": gw, "corrections": gc}
    if kind == "refit":
        w = state["weights"]
        w.grad = None
        sums, counts = polygenic_score(w, state["rows"], state["pitch"], state["flipped"],
                                       state["member"], case["people"])
        loss = (sums - state["target"]).square().mean()
        loss.backward()
        return {"sums": sums.detach(), "counts": counts, "grad": w.grad}
    if kind == "run":
        sums, counts = pipeline_run(state["context"], state["rows"])
        return {"sums": sums, "counts": counts}
    if kind == "project":
        V = case["variants"]
        with Projector(case["people"], case["axes"]) as pj:
            for b in range(case["blocks"]):
                s = slice(b * V, (b + 1) * V)
                pj.block(state["rows"][s], state["coeffs"][s], state["loadings"][s])
            return {"scores": pj.scores()}
    state["pgen"].decode(state["rows"], state["pitch"])
    return {"rows": state["rows"]}


def work(case):
    kind, P, V = case["kind"], case["people"], case["variants"]
    bpv = (P + 3) // 4
    if kind == "score":
        n, K = max(1, int(P * case["keep"])), case["scores"]
        cells = V * K * _share(case)
        return {"bytes": V * bpv + 8 * cells + 12 * n * K, "flops": 2 * n * cells}
    if kind == "backward":
        n, K = max(1, int(P * case["keep"])), case["scores"]
        return {"bytes": V * bpv + 4 * n * K + 8 * V * K, "flops": 2 * n * V * K}
    if kind == "refit":
        K = case["scores"]
        return {"bytes": 2 * V * bpv + 20 * P * K + 10 * V * K, "flops": 4 * P * V * K}
    if kind == "run":
        need, K = int(0.9 * V), case["scores"]
        cells = need * K * _share(case)
        return {"bytes": need * bpv + 8 * cells + 12 * P * K, "flops": 2 * P * cells}
    if kind == "project":
        n, K = case["blocks"] * V, case["axes"]
        return {"bytes": n * bpv + 12 * n + 4 * n * K + 8 * P * K, "flops": 2 * P * n * K}
    # .pgen: a record takes about half of the row that it becomes
    return {"bytes": 1.5 * V * case["repeats"] * bpv, "flops": 0}


# ---- the same in 64 bits, plain torch -----------------------------------------------


def _codes(rows, people):
    """Packed rows [n][>= bytes] on the GPU -> codes [n][people]."""
    b = rows[:, :(people + 3) // 4]
    return torch.stack([(b >> s) & 3 for s in (0, 2, 4, 6)], dim=-1).reshape(len(b), -1)[:, :people]


def _dosage_missing(codes):
    missing = codes == 1
    dosage = (codes >> 1) + (codes == 3).to(torch.uint8)
    return dosage.to(torch.float64), missing


def _chunks(variants, people):
    step = max(1, min(variants, (CHUNK // 2) // max(1, people)))
    return [slice(v, min(v + step, variants)) for v in range(0, variants, step)]


def _exact_scores(rows, people, w, flipped, member, keep=None):
    """sum over called genotypes of w * d (w * (2 - d) where flipped), and missing counts."""
    V, K = w.shape
    sums = torch.zeros(people, K, dtype=torch.float64, device=DEVICE)
    counts = torch.zeros(people, K, dtype=torch.float64, device=DEVICE)
    for s in _chunks(V, people):
        d, m = _dosage_missing(_codes(rows[s], people))
        m = m.to(torch.float64)
        mem = torch.from_numpy(member[s]).to(DEVICE)
        x = torch.from_numpy(w[s]).to(DEVICE).double() * mem
        f = torch.from_numpy(flipped[s]).to(DEVICE)
        signed, twice = torch.where(f, -x, x), torch.where(f, 2 * x, 0.0)
        sums += d.T @ signed + twice.sum(0) - m.T @ twice
        counts += m.T @ mem.double()
    counts = counts.round().to(torch.int32)
    if keep is not None:
        at = torch.from_numpy(keep.astype(np.int64)).to(DEVICE)
        sums, counts = sums[at], counts[at]
    return sums, counts


def _exact_grads(rows, people, grad, variants):
    """(sum over people of d * grad, minus the sum of grad over missing calls), [variants][K]."""
    gw, gc = [], []
    for s in _chunks(variants, people):
        d, m = _dosage_missing(_codes(rows[s], people))
        gw.append(d @ grad)
        gc.append(-(m.to(torch.float64) @ grad))
    return torch.cat(gw), torch.cat(gc)


def exact(case, seed):
    kind, P, V = case["kind"], case["people"], case["variants"]
    if kind == "pgen":
        return None                                    # bytes: compared with the start's
    d = _inputs(case, seed)
    if kind == "project":
        n, K = case["blocks"] * V, case["axes"]
        rows = torch.from_numpy(d["rows"]).to(DEVICE)
        out = torch.zeros(P, K, dtype=torch.float64, device=DEVICE)
        c = torch.from_numpy(d["coeffs"]).to(DEVICE).double()
        ld = torch.from_numpy(d["loadings"]).to(DEVICE).double()
        for s in _chunks(n, P):
            codes = _codes(rows[s], P)
            x = torch.zeros(codes.shape, dtype=torch.float64, device=DEVICE)
            for code, g in ((0, 0), (2, 1), (3, 2)):
                x += (codes == code) * c[s, g:g + 1]
            out += x.T @ ld[s]
        return {"scores": out.cpu().numpy()}
    if kind == "run":
        rows = torch.from_numpy(d["rows"]).to(DEVICE).view(V, -1)
        rows = rows[torch.from_numpy(d["required"].astype(np.int64)).to(DEVICE)]
        sums, counts = _exact_scores(rows, P, d["w"], d["flipped"], d["member"])
        return {"sums": sums.view(-1).cpu().numpy(),
                "counts": counts.view(-1).cpu().numpy().astype(np.uint32)}
    rows = d["rows"].view(V, d["pitch"])
    if kind == "score":
        sums, counts = _exact_scores(rows, P, d["w"], d["flipped"], d["member"], d["keep"])
        return {"sums": sums.view(-1), "counts": counts.view(-1)}
    grad = d["grad"].double()
    if kind == "backward":
        if d["keep"] is not None:
            at = torch.from_numpy(d["keep"].astype(np.int64)).to(DEVICE)
            grad = torch.zeros(P, grad.shape[1], dtype=torch.float64,
                               device=DEVICE).index_copy_(0, at, grad)
        gw, gc = _exact_grads(rows, P, grad, V)
        return {"weights": gw, "corrections": gc}
    sums, counts = _exact_scores(rows, P, d["w"], d["flipped"], d["member"])
    ds = 2 * (sums - grad) / sums.numel()
    gw, gc = _exact_grads(rows, P, ds, V)
    flipped = torch.from_numpy(d["flipped"]).to(DEVICE)
    g = torch.where(flipped, 2 * (ds.sum(0, keepdim=True) + gc) - gw, gw)
    g = torch.where(torch.from_numpy(d["member"]).to(DEVICE), g, 0.0)
    return {"sums": sums, "counts": counts, "grad": g}
