"""Timed workloads of the fitting path, through its public entry points.

A case is a dict: `op` (which call), `precision` ("fp64", the default of
GB300Admix and run_admixture, or "mixed", the default of k_sweep and of the
benchmark), the sizes I (individuals), J (two-SNP blocks) and K (ancestries),
and what the call takes besides.  Cohorts are synthetic, of the generator that
the benchmark configurations use (Q ~ Dirichlet(alpha), haplotype frequencies ~
Dirichlet(1,1,1,1), two haplotype copies per individual and block, 1% missing
calls), drawn here from the seed alone.
"""
import math
import os
import sys

import numpy as np
import torch

_PKG = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "haploadmixture.jl_gb300")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

MISS = 0.01
FLOOR = 1e-5      # the fit's floor on every entry of Q and P


def listed():
    return [
        # the smallest call: one log-likelihood from caller-owned device buffers, no allocation (a host
        # framework's own loop), at the CPU-runnable cohort size of the test configurations
        dict(name="loglik_small", op="loglik", precision="fp64", I=1000, J=1000, K=3),
        # a whole small fit from a random start, as run_admixture runs it with its default precision
        # (5 EM iterations, then QN iterations): launches, reductions and host steps count
        dict(name="fit_small", op="fit", precision="fp64", I=1000, J=1000, K=3, em=5, iters=6),
        # the K sweep's inner call: fits of several K on one decoded cohort at the same time
        dict(name="sweep_small", op="sweep", precision="mixed", I=5000, J=4000, K=5, kmin=2, em=5, iters=2),
        # plain FP64 outer iterations in mid-fit at a tenth of the 10,000 x 100,000 SNP configuration, K = 5
        dict(name="plain_mid", op="fit", precision="fp64", I=10000, J=5000, K=5, em=0, iters=2),
        # a large plain FP64 outer iteration at the benchmark's K = 8
        dict(name="plain_large", op="fit", precision="fp64", I=50000, J=4000, K=8, em=0, iters=1),
        # mixed outer iterations at the sweep's cohort size and its largest K
        dict(name="mixed_k10", op="fit", precision="mixed", I=20000, J=20000, K=10, em=0, iters=2),
        # the benchmark's shape (100,000 individuals, K = 8) on a fifth of its SNPs
        dict(name="mixed_large", op="fit", precision="mixed", I=100000, J=20000, K=8, em=0, iters=1),
        # the EM start of a mixed fit, ragged sizes
        dict(name="em_mixed", op="em", precision="mixed", I=50001, J=9999, K=6, em=5),
        # the reference's GPU runners on host arrays (update_q!, mixed; update_p!, FP64), odd sizes
        dict(name="accum_q_mixed", op="accum_q", precision="mixed", I=33331, J=6007, K=6),
        dict(name="accum_p_plain", op="accum_p", precision="fp64", I=7777, J=3001, K=4),
        # opening a cohort: upload of a .bed matrix from host memory, decode, census, double-missing counts
        dict(name="load", op="load", precision="mixed", I=50000, J=10000, K=8),
        # selection of ancestry-informative markers before a fit (run_admixture's sparsity branch)
        dict(name="skfr", op="skfr", precision="fp64", I=4000, J=10000, K=5, sparsity=500),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


# op -> (smallest, largest) I and J, and the most pairs I*J for FP64 and mixed
_RANGE = {
    "loglik": ((300, 20000), (300, 20000), 4e7, 4e7),
    "fit": ((500, 100000), (500, 40000), 1.2e8, 1.5e9),
    "em": ((500, 100000), (500, 40000), 1e8, 5e8),
    "sweep": ((500, 8000), (500, 8000), 1e7, 3e7),
    "accum_q": ((500, 60000), (500, 20000), 5e7, 3e8),
    "accum_p": ((500, 60000), (500, 20000), 5e7, 3e8),
    "load": ((1000, 60000), (1000, 20000), 4e8, 4e8),
    "skfr": ((500, 5000), (1000, 10000), 3e7, 3e7),
}


def draw(rng):
    op = rng.choice(["loglik", "fit", "fit", "fit", "em", "sweep", "accum_q", "accum_p", "load", "skfr"])
    precision = rng.choice(["fp64", "mixed"])
    (i0, i1), (j0, j1), most64, most = _RANGE[op]
    cap = most64 if precision == "fp64" else most
    K = rng.randint(2, 12)
    if op == "sweep":
        K = rng.randint(3, 6)
    if precision == "fp64":
        cap *= min(1.0, 110.0 / (K * K + 10 * K))     # the work of a pair grows like K^2
    I = _log(rng, i0, i1)
    J = _log(rng, j0, j1)
    if I * J > cap:
        J = max(j0, int(cap / I))
        I = max(i0, min(I, int(cap / J)))
    c = dict(op=op, precision=precision, I=I, J=J, K=K)
    if op == "fit":
        c.update(em=rng.choice([0, 0, 5]), iters=rng.randint(1, 2))
        if c["em"] and I * J > cap / 4:
            c["em"] = 0
    elif op == "sweep":
        c.update(kmin=2, em=5, iters=1)
    elif op == "em":
        c.update(em=rng.choice([1, 5]))
    elif op == "skfr":
        c.update(precision="fp64", sparsity=max(1, J // rng.randint(10, 40)))
    return c


# ------------------------------------------------------------------ inputs

def _params(case, seed):
    """True Q (I x K) and P (K x J x 4), and the state the call starts from
    (q: I x K, p: J x 4 x K, FP64; the library's column-major K x I, K x 4J)."""
    I, J, K = case["I"], case["J"], case["K"]
    rng = np.random.default_rng(seed)
    Q = rng.dirichlet(np.full(K, 0.5), size=I)
    P = rng.dirichlet(np.ones(4), size=(K, J))
    q, p = _start(I, J, K, rng)
    if case["op"] in ("fit", "accum_q", "accum_p", "loglik") and not case.get("em"):
        # in mid-fit: near the truth, entries down to the floor
        q = _floored(0.7 * Q + 0.3 * q)
        p = _floored((0.7 * P + 0.3 * p.reshape(J, 4, K).transpose(2, 0, 1))).transpose(1, 2, 0)
    return Q, P, np.ascontiguousarray(q), np.ascontiguousarray(p.reshape(J, 4, K))


def _start(I, J, K, rng):
    """The random start of a fit: uniform draws, normalised per individual and per (ancestry, block)."""
    q = rng.random((I, K))
    p = rng.random((J, 4, K))
    return q / q.sum(1, keepdims=True), p / p.sum(1, keepdims=True)


def _floored(x):
    """Rows with small entries set to the floor (last axis sums to 1)."""
    n = x.shape[-1]
    x = np.where(x < 0.02, 0.0, x)
    x = x / x.sum(-1, keepdims=True)
    return x * (1.0 - n * FLOOR) + FLOOR


def _bed(case, seed, Q, P):
    """The cohort's SNP-major .bed matrix (2J x ceil(I/4) bytes) on the GPU."""
    I, J, K = case["I"], case["J"], case["K"]
    dev = torch.device("cuda")
    gen = torch.Generator(device=dev)
    gen.manual_seed(seed)
    cq = torch.from_numpy(np.cumsum(Q, 1).astype(np.float32)).to(dev)
    cp = torch.from_numpy(np.cumsum(P, 2).astype(np.float32)).to(dev)
    code_of = torch.tensor([0, 2, 3], dtype=torch.uint8, device=dev)
    bps = (I + 3) // 4
    out = torch.empty((2 * J, bps), dtype=torch.uint8, device=dev)
    step = max(1, int(4e7 // I))
    for j0 in range(0, J, step):
        n = min(step, J - j0)
        a1 = torch.zeros((I, n), dtype=torch.uint8, device=dev)
        a2 = torch.zeros_like(a1)
        for _ in range(2):
            u = torch.rand((I, n), generator=gen, device=dev)
            z = torch.zeros((I, n), dtype=torch.int64, device=dev)
            for k in range(K - 1):
                z += u >= cq[:, k, None]
            u = torch.rand((I, n), generator=gen, device=dev)
            h = torch.zeros_like(a1)
            for t in range(3):
                h += u >= torch.gather(cp[:, j0:j0 + n, t], 0, z)
            a1 += h >> 1
            a2 += h & 1
        for s, a in ((0, a1), (1, a2)):
            c = code_of[a.long()]
            c[torch.rand((I, n), generator=gen, device=dev) < MISS] = 1
            c = torch.nn.functional.pad(c.t(), (0, 4 * bps - I)).reshape(n, bps, 4)
            out[2 * j0 + s:2 * (j0 + n):2] = c[..., 0] | (c[..., 1] << 2) | (c[..., 2] << 4) | (c[..., 3] << 6)
    return out


def prepare(case, seed):
    import haplo_gb300 as hx
    I, J, K = case["I"], case["J"], case["K"]
    Q, P, q, p = _params(case, seed)
    bed = _bed(case, seed, Q, P)
    torch.cuda.synchronize()
    s = dict(case=case, hx=hx, bps=bed.shape[1])
    op = case["op"]
    if op in ("load", "skfr"):
        s["bed"] = bed.cpu().numpy()
        return s
    dq, dp = torch.from_numpy(q).cuda(), torch.from_numpy(p).cuda()
    if op == "loglik":
        s.update(bed=bed, q=dq, p=dp, ll=torch.empty((), dtype=torch.float64, device="cuda"),
                 prec={"fp64": 0, "mixed": 1}[case["precision"]])
        torch.cuda.synchronize()
        return s
    s["d"] = d = hx.GB300Admix(bed.data_ptr(), I, J, K, bytes_per_snp=bed.shape[1], n_snp=2 * J,
                               precision=case["precision"], bed_on_device=True)
    if op in ("accum_q", "accum_p"):
        s.update(q=q.T, p=p.reshape(4 * J, K).T)
    elif op == "sweep":
        s["fits"] = []
        for k in range(case["kmin"], K + 1):
            a, b = (torch.from_numpy(np.ascontiguousarray(x)).cuda()
                    for x in _start(I, J, k, np.random.default_rng(seed + 1000 * k)))
            c = d if k == K else hx.GB300Admix.shared(d, k, precision=case["precision"])
            s["fits"].append((c, a, b))
    else:
        s.update(q=dq, p=dp)
    torch.cuda.synchronize()
    return s


# ------------------------------------------------------------------ the calls

def run(s):
    case, hx = s["case"], s["hx"]
    I, J, K, op = case["I"], case["J"], case["K"], case["op"]
    if op == "loglik":
        st = hx.load().hx_loglikelihood_noalloc(s["bed"].data_ptr(), s["bps"], I, J, K, s["q"].data_ptr(),
                                                s["p"].data_ptr(), s["prec"], s["ll"].data_ptr(),
                                                torch.cuda.current_stream().cuda_stream)
        if st:
            raise RuntimeError("hx_loglikelihood_noalloc: status %d" % st)
        return s["ll"]
    if op == "load":
        d = hx.GB300Admix(s["bed"], I, J, K, bytes_per_snp=s["bps"], n_snp=2 * J, precision=case["precision"])
        out = d.census(), d.double_missing()
        d.close()
        return out
    if op == "skfr":
        return hx.skfr.select_aims(s["bed"], I, K, case["sparsity"])
    if op == "sweep":
        for c, q, p in s["fits"]:
            c.set_qp_device(q.data_ptr(), p.data_ptr())
        infos = hx.sweep.fit_many([c for c, _, _ in s["fits"]], n_iter=case["iters"], rtol=0.0,
                                  em_iters=case["em"])
        return [(i["ll"], i["iters"], c.get_qp()) for i, (c, _, _) in zip(infos, s["fits"])]
    d = s["d"]
    if op == "accum_q":
        return d.update_q_accum(s["q"], s["p"])
    if op == "accum_p":
        return d.update_p_accum(s["q"], s["p"])
    d.set_qp_device(s["q"].data_ptr(), s["p"].data_ptr())
    if op == "em":
        d.init_em(case["em"])
        return d.get_qp(), d.ll_new
    info = d.fit(n_iter=case["iters"], rtol=0.0, em_iters=case["em"])
    return d.get_qp(), info["ll"]


# ------------------------------------------------------------------ floors

def work(case):
    """Bytes and operations of one pass that the path cannot do without: a
    pass over all pairs reads each pair's class (4 bits) once, Q and P once,
    and writes its sums once; per pair 8K operations for the four mixed
    haplotype frequencies, 8K per gradient and 4K(K+1) per Hessian triangle."""
    I, J, op = case["I"], case["J"], case["op"]
    bed = 2.0 * J * ((I + 3) // 4)
    pairs = float(I) * J
    if op == "load":
        return {"bytes": 2 * bed, "flops": 0.0}
    if op == "skfr":
        return {"bytes": bed, "flops": 2.0 * pairs * 2 * case["K"]}
    b = f = 0.0
    for K in range(case.get("kmin", case["K"]), case["K"] + 1):
        x = 8.0 * K * (I + 4 * J)
        hq, hp = 4.0 * K * (K + 1) * I, 16.0 * K * (K + 1) * J
        ll, grad, hess = 8.0 * K, 16.0 * K, 16.0 * K + 4.0 * K * (K + 1)
        if op == "loglik":
            b, f = b + bed + x, f + pairs * ll
        elif op == "accum_q":
            b, f = b + bed + x + 2 * hq + 8.0 * K * I, f + pairs * hess
        elif op == "accum_p":
            b, f = b + bed + x + 2 * hp + 32.0 * K * J, f + pairs * hess
        else:
            em, it = case["em"], case.get("iters", 0)
            b += em * (2 * bed + 2 * x) + bed + it * (6 * bed + 2 * (hq + hp) + 8 * x)
            f += pairs * (em * 2 * grad + ll + it * (4 * hess + 2 * ll))
    return {"bytes": b, "flops": f}


# ------------------------------------------------------------------ 64-bit values

# carrier sets of the two haplotype copies for each class (raw codes c1 + 4 c2 of the block's SNPs);
# haplotype h = 2 * allele(SNP 1) + allele(SNP 2).  The double heterozygote (both phases) and the
# double-missing class are treated apart.
def _sets():
    m = np.zeros((2, 16, 4))
    first = {0: (0,), 1: (0, 1), 2: (0,), 3: (1,)}
    second = {0: (0,), 1: (0, 1), 2: (1,), 3: (1,)}
    for c1 in range(4):
        for c2 in range(4):
            if (c1, c2) in ((1, 1), (2, 2)):
                continue
            for copy, of in ((0, first), (1, second)):
                for a in of[c1]:
                    for b in of[c2]:
                        m[copy, c1 + 4 * c2, 2 * a + b] = 1.0
    return m


def _blocks(bed, I, j0, n):
    """Class (c1 + 4 c2) of every pair, I x n."""
    b = bed[2 * j0:2 * (j0 + n)]
    c = torch.stack([(b >> (2 * r)) & 3 for r in range(4)], -1).reshape(n, 2, -1)[:, :, :I]
    return (c[:, 0] + 4 * c[:, 1]).long().t().contiguous()


def _chunks(bed, I, J, q, p):
    """For chunks of blocks: j0, n, p (n x 4 x K), qp and U = c / qp (I x n x 4) and log L summed."""
    m = torch.from_numpy(_sets()).cuda()
    K = q.shape[1]
    step = max(1, int(1.2e7 // I))
    for j0 in range(0, J, step):
        n = min(step, J - j0)
        nib = _blocks(bed, I, j0, n)
        pj = p[j0:j0 + n]
        qp = (q @ pj.reshape(4 * n, K).t()).reshape(I, n, 4)
        m1, m2 = m[0][nib], m[1][nib]
        hh, mm = nib == 10, nib == 5
        one = torch.ones((), dtype=torch.float64, device="cuda")
        F1 = torch.where(hh, qp[..., 0] * qp[..., 3] + qp[..., 1] * qp[..., 2], (m1 * qp).sum(-1))
        F1 = torch.where(mm, one, F1)
        F2 = torch.where(hh | mm, one, (m2 * qp).sum(-1))
        U = m1 / F1[..., None] + m2 / F2[..., None]
        U = torch.where(hh[..., None], qp.flip(-1) / F1[..., None], U)
        yield j0, n, pj, qp, U, torch.log(F1 * F2).sum(), mm


def _gradients(bed, I, J, q, p):
    gq, gp, ll = torch.zeros_like(q), torch.zeros_like(p), 0.0
    for j0, n, pj, qp, U, l, _ in _chunks(bed, I, J, q, p):
        gq += U.reshape(I, 4 * n) @ pj.reshape(4 * n, -1)
        gp[j0:j0 + n] = (U.reshape(I, 4 * n).t() @ q).reshape(n, 4, -1)
        ll = ll + l
    return gq, gp, ll


def _project(x):
    """Euclidean projection of the last axis onto {x >= FLOOR, sum x = 1}."""
    n = x.shape[-1]
    y = x - FLOOR
    total = 1.0 - n * FLOOR
    s = torch.sort(y, -1, descending=True).values
    t = (torch.cumsum(s, -1) - total) / torch.arange(1, n + 1, dtype=x.dtype, device=x.device)
    r = (s > t).sum(-1, keepdim=True).clamp(min=1)
    return torch.clamp(y - torch.gather(t, -1, r - 1), min=0.0) + FLOOR


def exact(case, seed):
    op, I, J, K = case["op"], case["I"], case["J"], case["K"]
    if op not in ("loglik", "accum_q", "accum_p", "em"):
        return None
    Q, P, q, p = _params(case, seed)
    bed = _bed(case, seed, Q, P)
    q, p = torch.from_numpy(q).cuda(), torch.from_numpy(p).cuda()
    if op == "loglik":
        return sum(c[5] for c in _chunks(bed, I, J, q, p))
    if op == "em":
        dm = sum(c[6].sum(1) for c in _chunks(bed, I, J, q, p)).double()
        for _ in range(case["em"]):
            gq, gp, _ll = _gradients(bed, I, J, q, p)
            q = _project(q * gq / (2.0 * (J - dm))[:, None])
            p = p * gp
            p = _project((p / p.sum(1, keepdim=True)).transpose(1, 2)).transpose(1, 2).contiguous()
        ll = sum(c[5] for c in _chunks(bed, I, J, q, p))
        return (q.t(), p.reshape(4 * J, K).t()), float(ll)
    if op == "accum_q":
        pp = p[..., :, None] * p[..., None, :]
        X, z = torch.zeros((I, K * K), dtype=torch.float64, device="cuda"), torch.zeros_like(q)
        for j0, n, pj, qp, U, _, _ in _chunks(bed, I, J, q, p):
            z += U.reshape(I, 4 * n) @ pj.reshape(4 * n, K)
            X += (U / qp).reshape(I, 4 * n) @ pp[j0:j0 + n].reshape(4 * n, K * K)
        return X.reshape(I, K, K).permute(1, 2, 0), z.t()
    qq = (q[:, :, None] * q[:, None, :]).reshape(I, K * K)
    X = torch.empty((4 * J, K * K), dtype=torch.float64, device="cuda")
    z = torch.empty((4 * J, K), dtype=torch.float64, device="cuda")
    for j0, n, pj, qp, U, _, _ in _chunks(bed, I, J, q, p):
        z[4 * j0:4 * (j0 + n)] = U.reshape(I, 4 * n).t() @ q
        X[4 * j0:4 * (j0 + n)] = (U / qp).reshape(I, 4 * n).t() @ qq
    return X.reshape(4 * J, K, K).permute(1, 2, 0), z.t()
