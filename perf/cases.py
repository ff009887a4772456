"""Performance cases: what a user of this framework runs, by step of its pipeline.

A run reads a PLINK BED matrix onto the GPU (``bed``), initialises from a randomized SVD of
the centred genotypes (``svd``), fits by Adam-EM (``em``: one iteration, in each E-step
arithmetic; ``fit``: a whole call) or by the default SQP + quasi-Newton algorithm
(``brqn``: the gradient/Hessian passes and the per-row QPs of one block update), and scores
the model by its log-likelihood (``loglik``). Sizes are those of the repository's
benchmark, tests and profiles, or generic cohorts; sample and SNP counts of real cohorts are
whatever they are, so odd ones stand beside the round ones.

Cohorts are synthetic admixed genotypes made on the GPU from the seed alone.
"""
import math

import torch

from adamixture_b200 import ops
from adamixture_b200.model.br_qn_gpu import compute_grad_hess_P_gpu, compute_grad_hess_Q_gpu
from adamixture_b200.model.em_adam_gpu import loglikelihood_gpu, optimize_parameters_gpu

DEV = "cuda"
CHUNK = 1 << 27          # entries made or evaluated at a time
LR, BETA1, BETA2, EPS = 0.005, 0.80, 0.88, 1e-8
STEP = 20.0              # Adam step number of the timed iterations


def listed():
    return [
        # the demo cohort's shape (105 samples), a short whole Adam-EM fit: the smallest calls,
        # where launches, captures and allocations are what a user waits for
        {"name": "fit_demo", "kind": "fit", "N": 105, "M": 8451, "K": 7, "iters": 20},
        # the biobank configuration in the default arithmetic of its K
        {"name": "em_f16_biobank", "kind": "em", "prec": "f16", "N": 200_000, "M": 500_000, "K": 10},
        # a mid-size cohort as cohorts come: neither count is round
        {"name": "em_f16_ragged", "kind": "em", "prec": "f16", "N": 10_007, "M": 200_003, "K": 8},
        # a small K, where the default arithmetic is float32
        {"name": "em_f32", "kind": "em", "prec": "f32", "N": 20_000, "M": 100_000, "K": 6},
        # the reference's own arithmetic, at the benchmark's K
        {"name": "em_f64", "kind": "em", "prec": "f64", "N": 100_000, "M": 50_000, "K": 10},
        # the two genotype passes of one SVD power iteration, at the held-out cohort's size of
        # the warm-start configuration (rank 10 + 10), and on a small odd cohort (rank 16 + 10)
        {"name": "svd_large", "kind": "svd", "N": 100_000, "M": 300_000, "L": 20},
        {"name": "svd_small", "kind": "svd", "N": 1_003, "M": 40_011, "L": 26},
        # the score of a start or of a finished model (float64 h), and the check every few
        # iterations of a float32 or tensor-core fit (float32 h)
        {"name": "loglik_f64", "kind": "loglik", "prec": "f64", "N": 50_000, "M": 100_000, "K": 8},
        {"name": "loglik_f32", "kind": "loglik", "prec": "f32", "N": 100_000, "M": 100_000, "K": 10},
        # one SQP block update of Q and of P in the default algorithm: a reference panel
        # (about 2,500 samples), and a larger cohort at a larger K
        {"name": "brqn_panel", "kind": "brqn", "N": 2_504, "M": 100_003, "K": 7},
        {"name": "brqn_large", "kind": "brqn", "N": 20_000, "M": 50_000, "K": 10},
        # reading a cohort: BED rows to the packed layout, frequencies, per-sample counts
        {"name": "bed_load", "kind": "bed", "N": 50_003, "M": 100_001},
    ]


def _log_int(rng, lo, hi):
    v = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    return max(lo, min(hi, v))


def _shape(rng, n, m, most):
    """N and M over their ranges, at most `most` entries; round sizes now and then."""
    N, M = _log_int(rng, *n), _log_int(rng, *m)
    while N * M > most:
        N, M = max(n[0], int(N * 0.8)), max(m[0], int(M * 0.8))
    if rng.random() < 0.3:
        N, M = max(16, N // 16 * 16), max(16, M // 16 * 16)
    return N, M


def draw(rng):
    kind = rng.choice(["fit", "em", "em", "em", "svd", "svd", "loglik", "loglik", "brqn", "brqn", "bed"])
    c = {"kind": kind}
    if kind == "fit":
        c["N"], c["M"] = _shape(rng, (50, 1_000), (2_000, 20_000), 2e7)
        c["K"], c["iters"] = rng.randint(2, 9), rng.choice([10, 15, 20])
    elif kind == "em":
        c["prec"] = rng.choice(["f16", "f16", "f32", "f64"])
        c["N"], c["M"] = _shape(rng, (500, 200_000), (5_000, 500_000), 1e10 if c["prec"] == "f16" else 3e9)
        c["K"] = rng.randint(8, 16) if c["prec"] == "f16" else rng.randint(2, 7) if c["prec"] == "f32" else rng.randint(2, 16)
    elif kind == "svd":
        c["N"], c["M"] = _shape(rng, (200, 200_000), (5_000, 300_000), 1e10)
        c["L"] = max(20, rng.randint(2, 26) + 10)
    elif kind == "loglik":
        c["prec"] = rng.choice(["f64", "f32"])
        c["N"], c["M"] = _shape(rng, (500, 200_000), (5_000, 300_000), 1e10 if c["prec"] == "f32" else 5e9)
        c["K"] = rng.randint(2, 16)
    elif kind == "brqn":
        c["N"], c["M"] = _shape(rng, (200, 20_000), (5_000, 100_000), 5e8)
        c["K"] = rng.randint(2, 12)
    else:
        c["N"], c["M"] = _shape(rng, (200, 100_000), (5_000, 300_000), 5e9)
    return c


# ------------------------------------------------------------------------------ cohorts

def _generator(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(seed)
    return g


def _model(N, M, K, gen):
    """Ancestral frequencies (minor-allele, correlated across populations) and admixture
    proportions (a mixture of near-pure and admixed samples), float64."""
    f = 0.05 + 0.45 * torch.rand((M, 1), generator=gen, device=DEV, dtype=torch.float64)
    z = torch.log(f / (1 - f)) + 0.5 * torch.randn((M, K), generator=gen, device=DEV, dtype=torch.float64)
    P = torch.sigmoid(z).clamp_(1e-5, 1 - 1e-5)
    scale = torch.where(torch.rand((N, 1), generator=gen, device=DEV) < 0.7, 6.0, 1.0).to(torch.float64)
    Q = torch.softmax(scale * torch.randn((N, K), generator=gen, device=DEV, dtype=torch.float64), 1)
    Q = Q.clamp_(1e-5, 1 - 1e-5)
    return P, Q / Q.sum(1, keepdim=True)


def _rows(N):
    """SNPs made at a time: whole packed rows of 4."""
    return max(4, CHUNK // N // 4 * 4)


def _dosages(P, Q, gen):
    """The cohort's dosages 0, 1, 2 (3: missing, about 1.2 %), a block of SNPs at a time:
    yields (first SNP, uint8 [block, N])."""
    M, N = P.shape[0], Q.shape[0]
    P32, QT = P.float(), Q.float().T.contiguous()
    for j in range(0, M, _rows(N)):
        h = P32[j:j + _rows(N)] @ QT
        u = torch.rand(h.shape, generator=gen, device=DEV)
        g = (u < h * h).to(torch.uint8)
        g += u < h * (2.0 - h)
        miss = torch.randint(0, 256, h.shape, generator=gen, device=DEV, dtype=torch.uint8) < 3
        yield j, g.masked_fill_(miss, 3)


def _packed(P, Q, gen):
    """The packed matrix [ceil(M/4), N]: SNP j of sample i in bits 2 (j % 4) of byte
    (j / 4, i); unused bits of the last row are 0."""
    M, N = P.shape[0], Q.shape[0]
    G = torch.empty(((M + 3) // 4, N), dtype=torch.uint8, device=DEV)
    for j, g in _dosages(P, Q, gen):
        pad = -g.shape[0] % 4
        if pad:
            g = torch.cat([g, torch.zeros((pad, N), dtype=torch.uint8, device=DEV)])
        g = g.view(-1, 4, N)
        G[j // 4:j // 4 + g.shape[0]] = g[:, 0] | g[:, 1] << 2 | g[:, 2] << 4 | g[:, 3] << 6
    return G


def _blocks(G, M):
    """The packed matrix's dosages in blocks, uint8: for the 64-bit values."""
    N = G.shape[1]
    step = max(4, (CHUNK // 4) // N // 4 * 4)
    for j in range(0, M, step):
        w = G[j // 4:(min(M, j + step) + 3) // 4]
        g = torch.stack([w >> (2 * s) & 3 for s in range(4)], 1).reshape(-1, N)
        yield j, g[:min(M, j + step) - j]


def _start(P, Q, gen):
    """A point part of the way to the fit: what an iteration of a running fit starts from."""
    mean = P.mean(1, keepdim=True)
    P0 = (0.8 * P + 0.2 * mean + 0.02 * torch.randn(P.shape, generator=gen, device=DEV, dtype=torch.float64))
    Q0 = 0.85 * Q + 0.15 / Q.shape[1]
    return P0.clamp_(1e-5, 1 - 1e-5).contiguous(), (Q0 / Q0.sum(1, keepdim=True)).contiguous()


def _moments(shape, gen):
    m = 1e-3 * torch.randn(shape, generator=gen, device=DEV, dtype=torch.float64)
    v = 1e-6 * (0.5 + torch.rand(shape, generator=gen, device=DEV, dtype=torch.float64))
    return m, v


def _inputs(case, seed):
    """What a case's path is given, from the seed alone."""
    gen = _generator(seed)
    kind, N, M = case["kind"], case["N"], case["M"]
    if kind == "bed":
        P, Q = _model(N, M, 6, gen)
        bed = torch.empty((M, (N + 3) // 4), dtype=torch.uint8, device=DEV)
        code = torch.tensor([3, 2, 0, 1], dtype=torch.uint8, device=DEV)  # dosage -> BED code
        for j, g in _dosages(P, Q, gen):
            b = torch.zeros((g.shape[0], (N + 3) // 4 * 4), dtype=torch.uint8, device=DEV)
            b[:, :N] = torch.where(g == 0, code[0], torch.where(g == 1, code[1], torch.where(g == 2, code[2], code[3])))
            b = b.view(g.shape[0], -1, 4)
            bed[j:j + g.shape[0]] = b[..., 0] | b[..., 1] << 2 | b[..., 2] << 4 | b[..., 3] << 6
        return {"bed": bed}
    if kind == "svd":
        P, Q = _model(N, M, 6, gen)
        G = _packed(P, Q, gen)
        L = case["L"]
        f = (P @ Q.mean(0)).float()
        Y = torch.randn((M, L), generator=gen, device=DEV)
        B = torch.randn((N, L), generator=gen, device=DEV) / math.sqrt(N)
        return {"G": G, "f": f, "Y": Y, "B": B}
    P, Q = _model(N, M, case["K"], gen)
    G = _packed(P, Q, gen)
    P, Q = _start(P, Q, gen)
    s = {"G": G, "P": P, "Q": Q}
    if kind == "em":
        s["mP"], s["vP"] = _moments(P.shape, gen)
        s["mQ"], s["vQ"] = _moments(Q.shape, gen)
        miss = torch.zeros(N, dtype=torch.float64, device=DEV)
        for j in range(0, G.shape[0], 4096):
            w = G[j:j + 4096]
            w = w & w >> 1 & 0x55
            miss += sum((w >> (2 * b) & 1).sum(0, dtype=torch.int64) for b in range(4))
        s["q_bat"] = 2.0 * (M - miss)
    return s


def prepare(case, seed):
    s = _inputs(case, seed)
    kind = case["kind"]
    s["case"] = case
    if kind == "em":
        if case["prec"] != "f64":
            s["P32"], s["Q32"] = s["P"].float(), s["Q"].float()
        s["ws"] = ops.em_workspace(case["M"], case["N"], case["K"], case["prec"], torch.device(DEV))
    elif kind == "loglik" and case["prec"] == "f32":
        s["P"], s["Q"] = s["P"].float(), s["Q"].float()
    elif kind == "brqn":
        N, M, K = case["N"], case["M"], case["K"]
        z = lambda *d: torch.zeros(d, dtype=torch.float64, device=DEV)  # noqa: E731
        s["XtX_q"], s["Xtz_q"], s["XtX_p"], s["Xtz_p"] = z(N, K, K), z(N, K), z(M, K, K), z(M, K)
        _, _, vt = torch.linalg.svd(torch.ones((1, K), dtype=torch.float64), full_matrices=True)
        s["v_kk"] = vt.t().contiguous().to(DEV)
    return s


def run(s):
    c = s["case"]
    kind, M, N = c["kind"], c["M"], c["N"]
    if kind == "fit":
        P, Q = optimize_parameters_gpu(s["G"], s["P"], s["Q"], LR, BETA1, BETA2, EPS, c["iters"], 5, c["K"], M, N,
                                       0.5, 1e-4, 3, 0.1, torch.device(DEV), 8192, 256, precision="f64")
        return {"P": P, "Q": Q}
    if kind == "em":
        f64 = c["prec"] == "f64"
        ops.em_adam_iteration(s["G"], s["P"], s["Q"], None if f64 else s["P32"], None if f64 else s["Q32"], s["mP"],
                              s["vP"], s["mQ"], s["vQ"], s["q_bat"], M, STEP, LR, BETA1, BETA2, EPS, c["prec"], s["ws"])
        # the updated model in the E-step's own input type: what the next iteration sweeps
        return {"P": s["P"], "Q": s["Q"]} if f64 else {"P": s["P32"], "Q": s["Q32"]}
    if kind == "svd":
        Z = ops.rsvd_cols(s["G"], s["f"], s["Y"], M)
        Y = ops.rsvd_rows(s["G"], s["f"], s["B"], M)
        return {"Z": Z, "Y": Y}
    if kind == "loglik":
        if c["prec"] == "f64":
            return loglikelihood_gpu(s["G"], s["P"], s["Q"], M, N, 8192, torch.device(DEV), 256)
        return ops.loglik_device(s["G"], s["P"], s["Q"], M, "f32")
    if kind == "brqn":
        K = c["K"]
        compute_grad_hess_Q_gpu(s["G"], s["Q"], s["P"], s["XtX_q"], s["Xtz_q"], M)
        Q1 = ops.sqp_solve_q(s["XtX_q"], -s["Xtz_q"], s["Q"], s["v_kk"], N, K)
        compute_grad_hess_P_gpu(s["G"], s["Q"], s["P"], s["XtX_p"], s["Xtz_p"], M)
        P1 = ops.sqp_solve_p(s["XtX_p"], -s["Xtz_p"], s["P"], M, K)
        return {"XtX_q": s["XtX_q"], "Xtz_q": s["Xtz_q"], "Q1": Q1, "XtX_p": s["XtX_p"], "Xtz_p": s["Xtz_p"], "P1": P1}
    G = ops.bed_to_packed(s["bed"], N, M)
    return {"G": G, "f": ops.allele_frequency(G, M), "q_bat": ops.sample_counts(G, M)}


def work(case):
    kind, N, M = case["kind"], case["N"], case["M"]
    g = (M + 3) // 4 * N            # the packed matrix
    if kind == "bed":
        # BED in, packed out, and the packed matrix once for each of the two statistics' results
        return {"bytes": M * ((N + 3) // 4) + g + 4 * M + 8 * N, "flops": 0}
    if kind == "svd":
        L = case["L"]
        return {"bytes": 2 * g + 4 * M + 8 * L * (M + N), "flops": 4 * M * N * L}
    K = case["K"]
    pq = K * (M + N)
    if kind == "fit":
        n = case["iters"] + 1
        return {"bytes": n * g + 16 * pq, "flops": n * 8 * M * N * K}
    if kind == "em":
        # P, Q and the moments read and written (float64); the sweep's own inputs
        return {"bytes": g + 6 * 8 * pq + (0 if case["prec"] == "f64" else 8 * pq), "flops": 8 * M * N * K}
    if kind == "loglik":
        return {"bytes": g + (8 if case["prec"] == "f64" else 4) * pq, "flops": 2 * M * N * K}
    # the symmetric K x K sums of both sides (two terms on the Q side), h and the gradients
    return {"bytes": 2 * g + 8 * (M + N) * (K * K + 4 * K), "flops": M * N * (3 * K * (K + 1) + 10 * K)}


# ------------------------------------------------------------------------------ 64-bit values

def _weights(g):
    """(g, 2 - g) as float64, both 0 where missing."""
    seen = g != 3
    gd = g.double() * seen
    return gd, 2.0 * seen - gd


def _stats(G, P, Q, M):
    A, B, T = torch.empty_like(P), torch.empty_like(P), torch.zeros_like(Q)
    for j, g in _blocks(G, M):
        p = P[j:j + g.shape[0]]
        h = (p @ Q.T).clamp_(1e-5, 1 - 1e-5)
        a, b = _weights(g)
        a /= h
        b /= 1.0 - h
        A[j:j + g.shape[0]] = a @ Q
        B[j:j + g.shape[0]] = b @ Q
        T += a.T @ p + b.T @ (1.0 - p)
    return A, B, T


def _adam(s, t, M):
    """One Adam-EM iteration in place on s (P, Q, mP, vP, mQ, vQ, q_bat)."""
    P, Q = s["P"], s["Q"]
    A, B, T = _stats(s["G"], P, Q, M)
    P_em = P * A / ((A - B) * P + B).clamp(min=1e-5)
    Q_em = Q * T / s["q_bat"].clamp(min=1e-5)[:, None]
    Q_em /= Q_em.sum(1, keepdim=True).clamp(min=1e-5)
    for x, target, m, v in ((P, P_em, s["mP"], s["vP"]), (Q, Q_em, s["mQ"], s["vQ"])):
        d = target - x
        m.mul_(BETA1).add_(d, alpha=1 - BETA1)
        v.mul_(BETA2).addcmul_(d, d, value=1 - BETA2)
        x += LR * (m / (1 - BETA1 ** t)) / ((v / (1 - BETA2 ** t)).sqrt() + EPS)
        x.clamp_(1e-5, 1 - 1e-5)
    Q /= Q.sum(1, keepdim=True)


def _loglik(G, P, Q, M):
    total = torch.zeros((), dtype=torch.float64, device=DEV)
    for j, g in _blocks(G, M):
        h = (P[j:j + g.shape[0]] @ Q.T).clamp_(1e-10, 1 - 1e-10)
        a, b = _weights(g)
        total += (a * torch.log(h)).sum() + (b * torch.log1p(-h)).sum()
    return total


def exact(case, seed):
    kind, M, N = case["kind"], case["M"], case["N"]
    if N * M > 5e10:   # well over 20 seconds in plain float64 tensor code
        return None
    s = _inputs(case, seed)
    if kind == "bed":
        bed = s["bed"]
        cnt, tot = torch.zeros(N, dtype=torch.float64, device=DEV), []
        for j in range(0, M, _rows(N)):
            b = bed[j:j + _rows(N)]
            c = torch.stack([b >> (2 * q) & 3 for q in range(4)], 2).reshape(b.shape[0], -1)[:, :N]
            g = torch.where(c == 3, 0, torch.where(c == 2, 1, torch.where(c == 0, 2, 3))).to(torch.uint8)
            seen = g != 3
            cnt += seen.sum(0)
            tot.append(torch.stack([(g * seen).sum(1, dtype=torch.int64), seen.sum(1, dtype=torch.int64)]))
        tot = torch.cat(tot, 1).double()
        f = tot[0] / (2.0 * tot[1]).clamp(min=1)
        if bool(tot[0].sum() / (2.0 * tot[1].sum()) >= 0.5):
            f = 1.0 - f
        return {"G": None, "f": f, "q_bat": 2.0 * cnt}
    if kind == "svd":
        G, f2 = s["G"], 2.0 * s["f"].double()
        Yin, B = s["Y"].double(), s["B"].double()
        Z, Y = torch.zeros_like(B), torch.empty_like(Yin)
        for j, g in _blocks(G, M):
            e = slice(j, j + g.shape[0])
            x = (g.double() - f2[e, None]).masked_fill_(g == 3, 0.0)
            Z += x.T @ Yin[e]
            Y[e] = x @ B
        return {"Z": Z, "Y": Y}
    G, P, Q = s["G"], s["P"], s["Q"]
    if kind == "loglik":
        if case["prec"] == "f32":
            P, Q = P.float().double(), Q.float().double()
        return _loglik(G, P, Q, M)
    if kind == "em":
        _adam(s, STEP, M)
        return {"P": P, "Q": Q}
    if kind == "fit":
        for x, m, v in (("P", "mP", "vP"), ("Q", "mQ", "vQ")):
            s[m], s[v] = torch.zeros_like(s[x]), torch.zeros_like(s[x])
        s["q_bat"] = torch.zeros(N, dtype=torch.float64, device=DEV)
        for _, g in _blocks(G, M):
            s["q_bat"] += 2.0 * (g != 3).sum(0)
        _adam(s, 1, M)
        best, kept = _loglik(G, P, Q, M), (P.clone(), Q.clone())
        for it in range(1, case["iters"] + 1):
            _adam(s, it + 1, M)
            if it % 5 == 0:
                L = _loglik(G, P, Q, M)
                if bool(L > best + 0.1):
                    best, kept = L, (P.clone(), Q.clone())
        return {"P": kept[0], "Q": kept[1]}
    K = case["K"]
    pairs = lambda x: (x[:, :, None] * x[:, None, :]).reshape(-1, K * K)  # noqa: E731
    Hq, gq = torch.zeros((N, K * K), dtype=torch.float64, device=DEV), torch.zeros_like(Q)
    Hp, gp = torch.empty((M, K * K), dtype=torch.float64, device=DEV), torch.empty_like(P)
    QQ = pairs(Q)
    for j, g in _blocks(G, M):
        e = slice(j, j + g.shape[0])
        p = P[e]
        h = (p @ Q.T).clamp_(1e-10, 1 - 1e-10)
        a, b = _weights(g)
        a /= h
        b /= 1.0 - h
        gq += a.T @ p + b.T @ (1.0 - p)
        gp[e] = (a - b) @ Q
        a /= h
        b /= 1.0 - h
        Hq += a.T @ pairs(p) + b.T @ pairs(1.0 - p)
        Hp[e] = (a + b) @ QQ
    return {"XtX_q": Hq.view(N, K, K), "Xtz_q": gq, "Q1": None, "XtX_p": Hp.view(M, K, K), "Xtz_p": gp, "P1": None}
