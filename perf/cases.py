"""Timed workloads of the EM and k-means engines, through their Python entry points.

A case names one call a program makes on data it already holds: training a
mixture, scoring rows with a trained one, a k-means run, a batch of fits.
`prepare` builds what such a program has in hand (rows on the device, the
handle, the initial mixture), `run` makes the call and returns everything it
produces, `exact` states the same results in plain 64-bit torch.

Parameters of fits whose precision option is "mixed" or "fp32" are returned as
float32, the precision those options compute in; the arrays are double only
because the interface shares them with the FP64 option, which stays float64.
"""
import math

import numpy as np
import torch

from fastem_gb300 import CudaBatchEM, CudaKMA, CudaMatrixEM, GaussianMixture

# the engines' limits and the sizes that the repository's workloads span
_KM_DIMS = (2, 4, 8, 16, 32, 64)
_BATCH_DIMS = (4, 7, 8, 16, 24, 32)


def listed():
    return [
        # the smallest fit: a few thousand rows, default precision; launches and host latency only
        dict(name="em_tiny", kind="em", n=3001, d=5, k=3, precision="mixed", sweeps=5, svd=True),
        # the parity workload: 100,000 rows in FP64, as the reference's double build runs it
        dict(name="em_fp64", kind="em", n=100000, d=8, k=10, precision="fp64", sweeps=10, svd=True),
        # an everyday fit with the default precision, ragged in every size
        dict(name="em_ordinary", kind="em", n=200003, d=24, k=21, precision="mixed", sweeps=5, svd=True),
        # a million rows at the headline's d and K
        dict(name="em_medium", kind="em", n=1 << 20, d=64, k=128, precision="mixed", sweeps=3, svd=True),
        # the headline workload: 8M rows
        dict(name="em_large", kind="em", n=1 << 23, d=64, k=128, precision="mixed", sweeps=3, svd=True),
        # more components than the tensor-core form takes: plain FP32
        dict(name="em_fp32", kind="em", n=250007, d=16, k=200, precision="fp32", sweeps=3, svd=False),
        # high-dimensional, condition 1e6 (the ill-conditioned workload with fewer rows)
        dict(name="em_wide", kind="em", n=3 << 17, d=256, k=64, precision="mixed", sweeps=2, svd=False),
        # the same path at an odd dimension and few rows
        dict(name="em_wide_ragged", kind="em", n=150001, d=99, k=23, precision="mixed", sweeps=3, svd=False),
        # a trained mixture applied to a new batch of host rows: posteriors and classes
        dict(name="score", kind="score", n=60000, d=32, k=32, precision="mixed"),
        # the k-means workload: 16M rows
        dict(name="km_large", kind="km", n=1 << 24, d=32, k=256, precision="mixed", iters=5, labels=False),
        # k-means in FP32 at another dimension, labels read back at the end
        dict(name="km_fp32", kind="km", n=1000003, d=16, k=100, precision="fp32", iters=8, labels=True),
        # many independent fits of uneven size in one batch
        dict(name="batch", kind="batch", fits=192, n_lo=2000, n_hi=200000, k_hi=32, precision="fp32", sweeps=8),
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(("mixed", "mixed", "fp64", "fp32", "wide", "score", "km_mixed", "km_fp32", "batch"))
    if kind == "mixed":
        d, k = _log_int(rng, 2, 64), _log_int(rng, 2, 128)
        return dict(kind="em", n=_log_int(rng, max(2000, 40 * k * d), 1 << 22), d=d, k=k, precision="mixed",
                    sweeps=rng.randint(2, 3), svd=rng.random() < 0.5)
    if kind == "fp64":
        d, k = rng.randint(2, 16), rng.randint(2, 16)
        return dict(kind="em", n=_log_int(rng, max(2000, 40 * k * d), 200000), d=d, k=k, precision="fp64",
                    sweeps=rng.randint(2, 8), svd=True)
    if kind == "fp32":
        d, k = _log_int(rng, 2, 40), _log_int(rng, 2, 256)
        return dict(kind="em", n=_log_int(rng, max(2000, 40 * k * d), max(500000, 40 * k * d)), d=d, k=k,
                    precision="fp32", sweeps=rng.randint(2, 3), svd=False)
    if kind == "wide":
        d, k = rng.randint(65, 256), _log_int(rng, 4, 64)
        return dict(kind="em", n=_log_int(rng, 16 * k * d, 1 << 19), d=d, k=k, precision="mixed",
                    sweeps=2, svd=False)
    if kind == "score":
        return dict(kind="score", n=_log_int(rng, 500, 200000), d=_log_int(rng, 2, 64), k=_log_int(rng, 2, 64),
                    precision=rng.choice(("mixed", "mixed", "fp32")))
    if kind == "km_mixed":
        return dict(kind="km", n=_log_int(rng, 10000, 1 << 23), d=32, k=_log_int(rng, 2, 256), precision="mixed",
                    iters=rng.randint(3, 8), labels=rng.random() < 0.5)
    if kind == "km_fp32":
        d = rng.choice(_KM_DIMS)
        return dict(kind="km", n=_log_int(rng, 10000, 2000000), d=d, k=_log_int(rng, 2, min(256, 9000 // d)),
                    precision="fp32", iters=rng.randint(3, 8), labels=rng.random() < 0.5)
    return dict(kind="batch", fits=_log_int(rng, 4, 160), n_lo=2000, n_hi=_log_int(rng, 20000, 200000),
                k_hi=rng.randint(4, 32), precision=rng.choice(("fp32", "mixed")), sweeps=rng.randint(3, 8))


# ------------------------------------------------------------------ inputs
def _mixture(rng, n, d, k, wide):
    """Weights, means, covariances to draw rows from, and the mixture that a
    k-means initialiser leaves for them: means a little off, covariances
    somewhat wide, equal weights."""
    w = np.maximum(rng.dirichlet(np.full(k, 2.0)), 0.3 / k)
    w /= w.sum()
    means = rng.normal(0.0, 10.0 if wide else 5.0, size=(k, d))
    q, r = np.linalg.qr(rng.standard_normal((k, d, d)))
    q *= np.sign(np.einsum("kii->ki", r))[:, None, :]
    if wide:
        lam = np.broadcast_to(np.logspace(-3.0, 3.0, d), (k, d))
    else:
        lam = np.exp(rng.uniform(math.log(0.1), math.log(10.0), size=(k, d)))
    covs = np.matmul(q * lam[:, None, :], q.transpose(0, 2, 1))
    covs = 0.5 * (covs + covs.transpose(0, 2, 1))
    root = q * np.sqrt(lam)[:, None, :]
    start_means = means + np.matmul(root, rng.normal(0.0, 0.2, size=(k, d, 1)))[:, :, 0]
    start = GaussianMixture(np.full(k, 1.0 / k), start_means, 1.25 * covs)
    return w, means, root, start


def _rows(gen, rng, n, w, means, root, dev):
    """n rows of the mixture on the device, in random order (float32)."""
    k, d = means.shape
    counts = rng.multinomial(n, w)
    x = torch.randn((n, d), generator=gen, device=dev)
    m = torch.tensor(means, dtype=torch.float32, device=dev)
    r = torch.tensor(root, dtype=torch.float32, device=dev)
    at = 0
    for j in range(k):
        c = int(counts[j])
        x[at:at + c] = torch.addmm(m[j], x[at:at + c], r[j].T)
        at += c
    return x[torch.randperm(n, generator=gen, device=dev)]


def _blobs(gen, rng, n, d, k, dev):
    """Isotropic blobs (sigma 1) of about equal size, and k rows to start from,
    drawn from a sample by the squared distance to those already drawn."""
    c = torch.tensor(rng.uniform(-20.0, 20.0, size=(k, d)), dtype=torch.float32, device=dev)
    x = torch.randn((n, d), generator=gen, device=dev)
    x += c[torch.randint(0, k, (n,), generator=gen, device=dev)]
    sample = x[:1 << 16]
    picked = [sample[0]]
    near = (sample - picked[0]).square().sum(1)
    for _ in range(k - 1):
        picked.append(sample[torch.multinomial(near, 1, generator=gen)[0]])
        near = torch.minimum(near, (sample - picked[-1]).square().sum(1))
    return x, torch.stack(picked).double().cpu().numpy()


def _batch_shapes(case):
    """Rows, dimension and components of every fit: a function of the case alone."""
    rng = np.random.default_rng(case["fits"])
    shapes = []
    for _ in range(case["fits"]):
        n = int(math.exp(rng.uniform(math.log(case["n_lo"]), math.log(case["n_hi"]))))
        d, k = int(rng.choice(_BATCH_DIMS)), int(rng.integers(2, case["k_hi"] + 1))
        shapes.append((n, d, max(2, min(k, n // (20 * d)))))   # rows enough for every covariance
    return shapes


def _inputs(case, seed):
    dev = torch.device("cuda", 0)
    gen = torch.Generator(device=dev)
    gen.manual_seed(seed)
    rng = np.random.default_rng(seed)
    if case["kind"] == "km":
        return _blobs(gen, rng, case["n"], case["d"], case["k"], dev)
    if case["kind"] == "batch":
        fits = []
        for n, d, k in _batch_shapes(case):
            w, means, root, start = _mixture(rng, n, d, k, False)
            fits.append((_rows(gen, rng, n, w, means, root, dev), start))
        return fits
    w, means, root, start = _mixture(rng, case["n"], case["d"], case["k"], case["d"] > 64)
    return _rows(gen, rng, case["n"], w, means, root, dev), start


def _reg(case):
    return 1e-6 if case["d"] > 64 else 0.0


def prepare(case, seed):
    got = _inputs(case, seed)
    state = dict(case=case)
    if case["kind"] == "em":
        x, state["start"] = got
        em = CudaMatrixEM(case["d"], case["n"], case["k"], precision=case["precision"])
        em.SetParameters(case["sweeps"], 0.0, 1e5, _reg(case))
        torch.cuda.synchronize()
        em.CopyDatasetDevice(x.data_ptr())
        state["em"] = em
    elif case["kind"] == "score":
        x, start = got
        em = CudaMatrixEM(case["d"], case["n"], case["k"], precision=case["precision"])
        em.SetMixture(start)
        em.InitDensities()
        state["em"], state["x"] = em, x.cpu().numpy()
    elif case["kind"] == "km":
        x, state["start"] = got
        km = CudaKMA(case["d"], case["n"], case["k"], precision=case["precision"])
        torch.cuda.synchronize()
        km.SetDatasetDevice(x.data_ptr())
        state["km"] = km
    else:
        shapes = [(x.shape[1], x.shape[0], g.GetComponentCount()) for x, g in got]
        em = CudaBatchEM(shapes, precision=case["precision"])
        em.SetParameters(case["sweeps"], 0.0, 1e5)
        em.CopyPacked(torch.cat([x.reshape(-1) for x, _ in got]).cpu().numpy())
        state["em"], state["start"] = em, [g for _, g in got]
    return state


# --------------------------------------------------------------------- run
def _held(case, a):
    """An array in the type of the precision it was computed in."""
    a = torch.from_numpy(np.ascontiguousarray(a))
    return a if case["precision"] == "fp64" else a.to(torch.float32)


def run(state):
    case = state["case"]
    if case["kind"] == "em":
        g = state["start"].copy()
        logl = state["em"].TrainNoCopy(g, svd=case["svd"])
        return dict(logl=logl, trace=_held(case, state["em"].logl_trace), weights=_held(case, g.weights),
                    means=_held(case, g.means), covs=_held(case, g.covs))
    if case["kind"] == "score":
        em = state["em"]
        em.CopyDataset(state["x"])
        logl = em.PrecomputeDensityMatrix()
        return dict(logl=logl, post=_held(case, em.Posteriors()), classes=em.RetrieveClasses())
    if case["kind"] == "km":
        km, cent = state["km"], state["start"].copy()
        km.Seed(1)   # an empty cluster is repaired by the same draws in every run
        fit = km.RunKMeans(cent, MaxIter=case["iters"] + 1)   # the reference's loop stops one short of MaxIter
        out = dict(fit=fit, centroids=cent)
        if case["labels"]:
            out["labels"] = km.Assignment()
        return out
    em = state["em"]
    for i, g in enumerate(state["start"]):
        em.SetMixture(i, g)
    status, iters, logl = em.TrainNoCopy()
    fits = [em.GetMixture(i) for i in range(em.nfits)]
    return dict(status=status, iters=iters, logl=_held(case, logl),
                weights=_held(case, np.concatenate([g.weights for g in fits])),
                means=_held(case, np.concatenate([g.means.reshape(-1) for g in fits])),
                covs=_held(case, np.concatenate([g.covs.reshape(-1) for g in fits])))


# -------------------------------------------------------------------- work
def _fit_work(n, d, k, sweeps):
    # per sweep the rows once, 2 n k d (d + 2) operations (triangular E-step product, means, upper covariance sums)
    return sweeps * 4.0 * n * d, sweeps * 2.0 * n * k * d * (d + 2)


def work(case):
    if case["kind"] == "em":
        b, f = _fit_work(case["n"], case["d"], case["k"], case["sweeps"])
        return dict(bytes=b + 16.0 * case["k"] * (case["d"] + 1) ** 2, flops=f)
    if case["kind"] == "score":
        n, d, k = case["n"], case["d"], case["k"]
        return dict(bytes=n * (4.0 * d + 8.0 * k + 4.0), flops=float(n) * k * d * (d + 1))
    if case["kind"] == "km":
        n, d, k = case["n"], case["d"], case["k"]
        return dict(bytes=case["iters"] * 4.0 * n * (d + 1), flops=case["iters"] * 2.0 * n * k * d)
    parts = [_fit_work(n, d, k, case["sweeps"]) for n, d, k in _batch_shapes(case)]
    return dict(bytes=sum(p[0] for p in parts), flops=sum(p[1] for p in parts))


# ------------------------------------------------------------------- exact
def _regularised(s, reg):
    """(1 - reg) S + reg tr(S) / d I, as the sweep regularises before it factorises."""
    if reg == 0.0:
        return s
    d = s.shape[-1]
    eye = torch.eye(d, dtype=s.dtype, device=s.device)
    return (1.0 - reg) * s + reg * torch.einsum("kii->k", s)[:, None, None] / d * eye


def _densities(x, pi, mu, s):
    """log(pi_j N(x; mu_j, S_j)) for every row and component (64 bits)."""
    n, d = x.shape
    low = torch.linalg.cholesky(s)
    inv = torch.linalg.solve_triangular(low, torch.eye(d, dtype=s.dtype, device=s.device).expand_as(low), upper=False)
    const = torch.log(pi) - 0.5 * d * math.log(2.0 * math.pi) - torch.log(torch.diagonal(low, dim1=1, dim2=2)).sum(1)
    out = torch.empty((n, len(pi)), dtype=torch.float64, device=x.device)
    for j in range(len(pi)):
        out[:, j] = const[j] - 0.5 * ((x - mu[j]) @ inv[j].T).square_().sum(1)
    return out


def _sweeps(x32, start, sweeps, reg):
    """EM sweeps in 64 bits: logL of each, and the parameters after the last."""
    dev, n, d = x32.device, x32.shape[0], x32.shape[1]
    pi, mu, s = (torch.tensor(a, dtype=torch.float64, device=dev) for a in (start.weights, start.means, start.covs))
    k = len(pi)
    s = _regularised(s, reg)
    step = max(1024, min(1 << 18, (1 << 30) // (8 * max(k, d))))
    trace = []
    for _ in range(sweeps):
        post = torch.empty((n, k), dtype=torch.float64, device=dev)
        logl = 0.0
        for a in range(0, n, step):
            lt = _densities(x32[a:a + step].double(), pi, mu, s)
            lse = torch.logsumexp(lt, 1)
            post[a:a + step] = torch.exp(lt - lse[:, None])
            logl += float(lse.sum())
        trace.append(logl)
        total = post.sum(0)
        sums = torch.zeros_like(mu)
        for a in range(0, n, step):
            sums += post[a:a + step].T @ x32[a:a + step].double()
        pi, mu = total / n, sums / total[:, None]
        s = torch.zeros_like(s)
        for a in range(0, n, step):
            x = x32[a:a + step].double()
            for j in range(k):
                t = x - mu[j]
                s[j] += (t * post[a:a + step, j:j + 1]).T @ t
        s = _regularised(s / total[:, None, None], reg)
    return trace, pi, mu, s


def _cost(n, d, k, sweeps):
    return 4.0 * n * k * d * d * sweeps   # 64-bit operations of _sweeps


def exact(case, seed):
    if case["kind"] == "em":
        if _cost(case["n"], case["d"], case["k"], case["sweeps"]) > 1.4e13:
            return None
        x, start = _inputs(case, seed)
        trace, pi, mu, s = _sweeps(x, start, case["sweeps"], _reg(case))
        return dict(logl=trace[-1], trace=torch.tensor(trace, dtype=torch.float64), weights=pi, means=mu, covs=s)
    if case["kind"] == "score":
        x, start = _inputs(case, seed)
        p = [torch.tensor(a, dtype=torch.float64, device=x.device) for a in (start.weights, start.means, start.covs)]
        lt = _densities(x.double(), *p)
        lse = torch.logsumexp(lt, 1)
        return dict(logl=float(lse.sum()), post=torch.exp(lt - lse[:, None]), classes=None)
    if case["kind"] == "km":
        if 3.0 * case["n"] * case["k"] * case["d"] * case["iters"] > 8e11:
            return None
        x, start = _inputs(case, seed)
        k, cent = case["k"], torch.tensor(start, dtype=torch.float64, device=x.device)
        best, step = math.inf, max(1024, (1 << 27) // (k * 8))
        for _ in range(case["iters"]):
            sums, counts, fit = torch.zeros_like(cent), torch.zeros(k, dtype=torch.float64, device=x.device), 0.0
            for a in range(0, case["n"], step):
                xs = x[a:a + step].double()
                near = torch.cdist(xs, cent, compute_mode="donot_use_mm_for_euclid_dist").min(1)
                fit += float(near.values.square().sum())
                sums.index_add_(0, near.indices, xs)
                counts += torch.bincount(near.indices, minlength=k)
            if fit / case["n"] < best:
                best = fit / case["n"]
            if bool((counts == 0).any()):
                return None   # an empty cluster is repaired from the engine's own random stream
            cent = sums / counts[:, None]
        return dict(fit=best, centroids=cent, **(dict(labels=None) if case["labels"] else {}))
    fits = _inputs(case, seed)
    if sum(_cost(x.shape[0], x.shape[1], g.GetComponentCount(), case["sweeps"]) for x, g in fits) > 1.4e13:
        return None
    got = [_sweeps(x, g, case["sweeps"], 0.0) for x, g in fits]
    return dict(status=None, iters=None,
                logl=torch.tensor([t[0][-1] for t in got], dtype=torch.float64),
                weights=torch.cat([t[1] for t in got]), means=torch.cat([t[2].reshape(-1) for t in got]),
                covs=torch.cat([t[3].reshape(-1) for t in got]))
