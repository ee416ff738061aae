"""Performance cases of the sampler's per-iteration path on one B200.

Four kinds of work, each through the entry points that a program calls:

  sweep   Gibbs sweeps through the device back-end (CudaKernel over the C ABI), the loop body of the
          sampler and of an adapter that derives from the reference's cudaKernel: parameter draws from
          the statistics, cluster labels, sub-cluster labels with their statistics, split and merge
          ratios; the labels and sub-labels are read back at the end of the pass.  NIW or Dirichlet
          prior.  The points are uploaded from device memory, and labels are read into pinned memory.
  score   the statistics and every split / merge log ratio of a labelling that the program brings
          (a warm start from another clustering): the labels go in from the host, the numbers come out.
  fit     dp_parallel: the whole call from host points (context, upload, every iteration, labels).
  batch   BatchSampler: one iteration of many uneven data sets together, and their labels.

A case is a dict of plain values.  Data are seeded draws of the generative models of the
configurations (Gaussian mixtures with covariances A A^T / D + 0.5 I; multinomial documents).
"""
import ctypes
import math

import numpy as np
import torch

from dpmmsubclusters_gpu_b200 import api, capi
from dpmmsubclusters_gpu_b200.screen import load_params


def listed():
    return [
        # the smallest data set anybody runs: launches and host latency are all there is
        dict(name="sweep_n2k_d2", kind="sweep", prior="gauss", n=2000, d=2, k=3, sd=8.0, sweeps=1, screen=False,
             final=False, fp32=False),
        # low-dimensional features (colour and position, flow cytometry), an odd number of points
        dict(name="sweep_n1m_d7", kind="sweep", prior="gauss", n=1000003, d=7, k=30, sd=6.0, sweeps=2, screen=False,
             final=False, fp32=False),
        # the million-point D = 32 configuration in its steady state: separated clusters
        dict(name="sweep_n1m_d32", kind="sweep", prior="gauss", n=1000000, d=32, k=20, sd=11.5, sweeps=2, screen=False,
             final=False, fp32=False),
        # the same size while the clusters still overlap (first iterations): every cluster matters to every point
        dict(name="overlap_n1m_d32", kind="sweep", prior="gauss", n=1000000, d=32, k=20, sd=0.4, sweeps=2,
             screen=False, final=False, fp32=False),
        # overlapping clusters at a ragged size and a dimension that is padded
        dict(name="overlap_n300k_d50", kind="sweep", prior="gauss", n=300001, d=50, k=64, sd=0.3, sweeps=2,
             screen=False, final=False, fp32=False),
        # the headline size: ten million points, D = 64, 100 clusters, the learned screen in front of the
        # merge ratios; labels read every fourth sweep
        dict(name="sweep_n10m_d64", kind="sweep", prior="gauss", n=10000000, d=64, k=100, sd=5.0, sweeps=4, screen=True,
             final=False, fp32=False),
        # high-dimensional features (embeddings after PCA): the widest Gaussian kernels
        dict(name="sweep_n100k_d100", kind="sweep", prior="gauss", n=100003, d=100, k=12, sd=3.0, sweeps=1, screen=False,
             final=False, fp32=False),
        # count vectors over a vocabulary of 1000
        dict(name="sweep_mult_n200k_d1000", kind="sweep", prior="mult", n=200000, d=1000, k=50, sd=0.1, sweeps=1,
             screen=False, final=False, fp32=False),
        # a small document collection with a short vocabulary
        dict(name="sweep_mult_n20k_d60", kind="sweep", prior="mult", n=20011, d=60, k=12, sd=0.2, sweeps=1,
             screen=False, final=False, fp32=False),
        # a labelling brought from elsewhere: its statistics and every split and merge ratio
        dict(name="score_n300k_d64", kind="score", n=300000, d=64, k=48, sd=2.0),
        # the whole call on the plain two-dimensional configuration
        dict(name="fit_n100k_d2", kind="fit", n=100000, d=2, k=2, sd=50.0, iters=40),
        # sixteen uneven data sets advanced together, one iteration at a time
        dict(name="batch_16_sets", kind="batch", sets=16, n_lo=1000, n_hi=60000, warm=40),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["sweep", "sweep", "sweep", "sweep", "overlap", "overlap", "mult", "mult", "score", "fit", "batch"])
    if kind in ("sweep", "overlap"):
        d = _log_int(rng, 2, 128)
        dp = 4
        while dp < d:
            dp *= 2
        k = _log_int(rng, 2, 100 if d <= 64 else 20)
        # bounded by what the largest listed cases cost: bytes of points, and for overlapping clusters
        # the dense N x K x D^2 work as well
        hi = min(4e6, 1.6e8 / dp, 4e5 if d > 64 else 4e6)
        if kind == "overlap":
            hi = min(hi, 1e11 / (k * dp * dp))
        n = _log_int(rng, 1500, max(3000, hi))
        return dict(kind="sweep", prior="gauss", n=n, d=d, k=k, sd=rng.choice([5.0, 8.0]) if kind == "sweep" else 0.3,
                    sweeps=rng.choice([1, 2, 4]), screen=k >= 40 and rng.random() < 0.5, final=rng.random() < 0.1,
                    fp32=rng.random() < 0.1 and n * k * dp * dp < 3e10)
    if kind == "mult":
        d = _log_int(rng, 20, 2000)
        return dict(kind="sweep", prior="mult", n=_log_int(rng, 1500, min(4e5, 2e8 / d)), d=d, k=_log_int(rng, 2, 80),
                    sd=rng.choice([0.1, 0.3]), sweeps=rng.choice([1, 2]), screen=False, final=rng.random() < 0.1,
                    fp32=False)
    if kind == "score":
        d = _log_int(rng, 2, 64)
        return dict(kind="score", n=_log_int(rng, 5000, 1.5e7 / d), d=d, k=_log_int(rng, 2, 48), sd=rng.choice([1.0, 4.0]))
    if kind == "fit":
        d = _log_int(rng, 2, 16)
        return dict(kind="fit", n=_log_int(rng, 2000, 1e6 / d), d=d, k=rng.randint(2, 8), sd=40.0,
                    iters=rng.randint(20, 45))
    return dict(kind="batch", sets=rng.randint(4, 16), n_lo=1000, n_hi=_log_int(rng, 4000, 60000), warm=40)


# ----------------------------------------------------------------------------- data
def _gauss_model(case, g):
    """Weights, means and covariance factors of the mixture, drawn on the CPU from the generator."""
    d, k = case["d"], case["k"]
    w = 0.5 + torch.rand(k, generator=g, dtype=torch.float64)
    mu = torch.randn(k, d, generator=g, dtype=torch.float64) * case["sd"]
    a = torch.randn(k, d, d, generator=g, dtype=torch.float64)
    cov = a @ a.transpose(1, 2) / d + 0.5 * torch.eye(d, dtype=torch.float64)
    return w / w.sum(), mu, torch.linalg.cholesky(cov)


def _gauss_points(case, seed):
    """float32 points (N x D, on the GPU) and the cluster (0-based) that each was drawn from."""
    g = torch.Generator().manual_seed(int(seed))
    w, mu, chol = _gauss_model(case, g)
    n, d, k = case["n"], case["d"], case["k"]
    gd = torch.Generator(device="cuda").manual_seed(int(seed) + 1)
    z = torch.multinomial(w.float().cuda(), n, replacement=True, generator=gd)
    x = torch.randn(n, d, device="cuda", generator=gd)
    mu32, chol32 = mu.float().cuda(), chol.float().cuda()
    order = torch.argsort(z, stable=True)
    starts = [0] + torch.cumsum(torch.bincount(z, minlength=k), 0).tolist()
    for c in range(k):
        rows = order[starts[c]:starts[c + 1]]
        x[rows] = x[rows] @ chol32[c].T + mu32[c]
    return x, z


def _mult_points(case, seed):
    """Counts (float32 N x D, on the GPU) of documents of about 200 words (60 below 100 categories), and
    their components."""
    n, d, k = case["n"], case["d"], case["k"]
    rng = np.random.default_rng(int(seed))
    theta = torch.from_numpy(rng.dirichlet(np.full(d, case["sd"]), size=k) + 1e-9).float().cuda()
    w = torch.from_numpy(rng.dirichlet(np.full(k, 4.0))).float().cuda()
    g = torch.Generator(device="cuda").manual_seed(int(seed) + 1)
    z = torch.multinomial(w, n, replacement=True, generator=g)
    mean = 200.0 if d >= 100 else 60.0
    lens = torch.poisson(torch.full((n,), mean, device="cuda"), generator=g).long()
    top = int(lens.max().item())
    cdf = torch.cumsum(theta.double(), 1)
    cdf = (cdf / cdf[:, -1:]).float()
    x = torch.zeros(n, d, device="cuda")
    for a in range(0, n, 100000):
        b = min(n, a + 100000)
        u = torch.rand(b - a, top, device="cuda", generator=g)
        keep = (torch.arange(top, device="cuda")[None, :] < lens[a:b, None]).float()
        cat = torch.empty(b - a, top, dtype=torch.long, device="cuda")
        for c in range(k):
            rows = (z[a:b] == c).nonzero()[:, 0]
            if rows.numel():
                cat[rows] = torch.searchsorted(cdf[c], u[rows].reshape(-1)).reshape(-1, top).clamp_(max=d - 1)
        x[a:b].scatter_add_(1, cat, keep)
    return x, z


def _niw(d):
    return api.niw_hyperparams(1.0, np.zeros(d), d + 3.0, np.eye(d))


ALPHA = 10.0


# ----------------------------------------------------------------------------- prepare
def _backend(case, x, prior):
    """A back-end context with the points of a device tensor."""
    L = capi.lib()
    k = api.CudaKernel(prior)
    k.N, k.D = x.shape
    d = capi.dpmm_desc()
    d.n_points, d.dim, d.prior_type, d.seed = k.N, k.D, int(prior), 1234
    d.loglik_mode = capi.LL_FP32 if case.get("fp32") else capi.LL_AUTO
    h = ctypes.c_void_p()
    capi.check(L.dpmm_create(ctypes.byref(d), ctypes.byref(h)))
    k.ctx = h
    torch.cuda.synchronize()   # the points are made on torch's stream
    capi.check(L.dpmm_upload_points_f32(k.ctx, ctypes.cast(x.data_ptr(), ctypes.POINTER(ctypes.c_float))))
    return k


def _pinned(n):
    return torch.empty(n, dtype=torch.int32, pin_memory=True)


def _prepare_sweep(case, seed):
    gauss = case["prior"] == "gauss"
    prior = api.prior_type.Gaussian if gauss else api.prior_type.Multinomial
    x, z = _gauss_points(case, seed) if gauss else _mult_points(case, seed)
    k = _backend(case, x, prior)
    k.set_prior(_niw(case["d"]) if gauss else api.multinomial_hyper(np.ones(case["d"])))
    if case["screen"]:
        k.screen_set_params(load_params())
    rng = np.random.default_rng(int(seed) + 2)
    k.set_labels((z + 1).int().cpu().numpy())
    k.set_sub_labels(rng.integers(1, 3, size=case["n"], dtype=np.int32))
    del x, z
    torch.cuda.empty_cache()
    K = case["k"]
    if gauss and case["d"] > 64:
        _set_given_params(k, case, seed)
    k.create_sufficient_statistics(np.arange(K))
    s = dict(case=case, k=k, step=0, counts=k.statistics_counts(np.arange(K)), seed=int(seed),
             labels=_pinned(case["n"]), sub=_pinned(case["n"]), all=np.arange(K, dtype=np.int32),
             eligible=np.ones(K, np.uint8), final=case["final"])
    for _ in range(3):   # from the generating labels to the sampler's own state
        _sweep(s, final=False)
    return s


def _set_given_params(k, case, seed):
    """Above 64 dimensions the parameters come from the host: those of the generating model, each cluster's
    two halves set apart along a random direction."""
    w, mu, chol = _gauss_model(case, torch.Generator().manual_seed(int(seed)))
    K, d = case["k"], case["d"]
    factor = torch.linalg.inv(chol).transpose(1, 2)   # sigma = L L^T: inv_sigma = W W^T with W = L^-T
    logdet = 2.0 * torch.log(torch.diagonal(chol, dim1=1, dim2=2)).sum(1)
    side = torch.from_numpy(np.random.default_rng(int(seed) + 3).normal(size=(K, d)) / math.sqrt(d))
    two = lambda t: torch.stack([t, t], 1).numpy()  # noqa: E731
    k.set_gaussian_params(mu.numpy(), factor.numpy(), logdet.numpy(), w.numpy(), torch.stack([mu + side, mu - side], 1).numpy(),
                          two(factor), two(logdet), np.full((K, 2), 0.5), factors=True)


def _sweep(s, final):
    """One iteration of the back-end: draws (where the device makes them: up to 64 dimensions), labels,
    sub-labels and statistics, split and merge ratios."""
    case, k = s["case"], s["k"]
    K, n = case["k"], case["n"]
    c = s["counts"].astype(np.float64)
    w = (c[:, 0] + ALPHA / K) / (n + ALPHA)
    lr = (c[:, 1:] + 0.5 * ALPHA) / (c[:, 1:].sum(1, keepdims=True) + ALPHA)
    s["step"] += 1
    lml = None
    if case["prior"] == "mult":
        lml = k.sample_multinomial_params(K, s["seed"], s["step"], lr)
    elif case["d"] <= 64:
        lml = k.sample_gaussian_params(K, s["seed"], s["step"], w, lr)
    k.create_clusters_labels(K, final)
    k.create_subclusters_labels(K)
    s["counts"] = k.statistics_counts(s["all"])
    slots, split = k.split_hastings(K, ALPHA)
    if case["screen"]:
        rows, scores = k.screen_select(K, capi.SCREEN_MERGE, ALPHA, s["eligible"], 16)
        i = s.setdefault("tri", np.triu_indices(K, 1))
        merge = k.merge_hastings_list(K, ALPHA, np.stack([i[0][rows], i[1][rows]], 1))
    else:
        rows = s["all"]
        merge = k.merge_hastings(K, ALPHA)
    return dict(lml=lml, slots=slots, split=split, merge=merge, rows=rows, counts=s["counts"])


def _run_sweep(s):
    for _ in range(s["case"]["sweeps"]):
        out = _sweep(s, s["final"])
    L, k = capi.lib(), s["k"]
    as_i32 = lambda t: ctypes.cast(t.data_ptr(), ctypes.POINTER(ctypes.c_int32))  # noqa: E731
    capi.check(L.dpmm_get_labels(k.ctx, as_i32(s["labels"])))
    capi.check(L.dpmm_get_sub_labels(k.ctx, as_i32(s["sub"])))
    out["labels"], out["sub"] = s["labels"], s["sub"]
    return out


def _score_inputs(case, seed):
    x, z = _gauss_points(case, seed)
    rng = np.random.default_rng(int(seed) + 2)
    lab = (z + 1).int().cpu().numpy()
    stray = rng.random(case["n"]) < 0.05   # an imperfect labelling
    lab[stray] = rng.integers(1, case["k"] + 1, size=int(stray.sum()), dtype=np.int32)
    return x, lab, rng.integers(1, 3, size=case["n"], dtype=np.int32)


def _prepare_score(case, seed):
    x, lab, sub = _score_inputs(case, seed)
    k = _backend(case, x, api.prior_type.Gaussian)
    k.set_prior(_niw(case["d"]))
    pl, ps = _pinned(case["n"]), _pinned(case["n"])
    pl.copy_(torch.from_numpy(lab))
    ps.copy_(torch.from_numpy(sub))
    return dict(case=case, k=k, labels=pl.numpy(), sub=ps.numpy(), all=np.arange(case["k"], dtype=np.int32), keep=(pl, ps))


def _run_score(s):
    k, K = s["k"], s["case"]["k"]
    k.set_labels(s["labels"])
    k.set_sub_labels(s["sub"])
    count, total, scatter = k.create_sufficient_statistics(s["all"])
    lml, split = k.split_hastings(K, ALPHA)
    return dict(count=count, total=total, scatter=scatter, lml=lml, split=split, merge=k.merge_hastings(K, ALPHA))


def _prepare_fit(case, seed):
    x, _ = _gauss_points(case, seed)
    return dict(case=case, x=np.ascontiguousarray(x.double().cpu().numpy()).T, seed=int(seed) % 100000 + 1)


def _table(weights, size):
    """The weights of however many clusters there are, as a table of the capacity."""
    out = np.zeros(size)
    out[:len(weights)] = weights
    return out


def _run_fit(s):
    c = s["case"]
    m = api.dp_parallel_sampling_class(c["n"], s["x"], s["seed"], api.prior_type.Gaussian)
    r = m.dp_parallel(_niw(c["d"]), 1.0, iters=c["iters"], init_clusters=1, verbose=False, burnout=5)
    return dict(labels=r.labels, weights=_table(r.weights, 256), clusters=r.cluster_count_history)


def _batch_shapes(case):
    """(N, D, K) of every data set: sizes spread over their logarithm, the four dimensions in turn."""
    m, lo, hi = case["sets"], math.log(case["n_lo"]), math.log(case["n_hi"])
    return [(int(math.exp(lo + (hi - lo) * i / max(1, m - 1))), (2, 8, 16, 64)[i * 7 % 4], 2 + i * 5 % 14) for i in range(m)]


def _prepare_batch(case, seed):
    data, hypers = [], []
    for i, (n, d, k) in enumerate(_batch_shapes(case)):
        x, _ = _gauss_points(dict(n=n, d=d, k=k, sd=6.0), int(seed) * 131 + i)
        data.append(x.double().cpu().numpy().T)
        hypers.append(_niw(d))
    b = api.BatchSampler(data, hypers, 5.0, iters=1 << 30, burnout=5)
    b.step(case["warm"])
    return dict(case=case, b=b)


def _run_batch(s):
    s["b"].step(1)
    infos = [s["b"].model_info(i) for i in range(s["case"]["sets"])]
    return dict(labels=[m.labels for m in infos], weights=[_table(m.weights, 64) for m in infos])


def prepare(case, seed):
    return dict(sweep=_prepare_sweep, score=_prepare_score, fit=_prepare_fit, batch=_prepare_batch)[case["kind"]](case, seed)


def run(state):
    kind = state["case"]["kind"]
    return dict(sweep=_run_sweep, score=_run_score, fit=_run_fit, batch=_run_batch)[kind](state)


# ----------------------------------------------------------------------------- work
def _gauss_sweep_work(n, d, k, overlapped):
    """One Gaussian iteration: the points once, labels and sub-labels out; the log-likelihoods of the
    clusters that matter to a point (all of them while they overlap, else its own), two sub-clusters, the
    upper triangle of the scatter, and a factorisation per slot."""
    flops = n * d * d * (2.0 * (k if overlapped else 1) + 4.0 + 1.0) + 3 * k * d ** 3
    return 4.0 * n * d + 8.0 * n, flops


def work(case):
    kind = case["kind"]
    if kind == "sweep" and case["prior"] == "gauss":
        n, d, k = case["n"], case["d"], case["k"]
        b, f = _gauss_sweep_work(n, d, k, case["sd"] < 1)
        pairs = 16 if case["screen"] else k * (k - 1) / 2
        return {"bytes": case["sweeps"] * b, "flops": case["sweeps"] * (f + pairs * d ** 3 / 3.0)}
    if kind == "sweep":
        n, d, k = case["n"], case["d"], case["k"]
        return {"bytes": case["sweeps"] * (2.0 * n * d + 8.0 * n), "flops": case["sweeps"] * n * d * (2.0 * k + 4.0 + 1.0)}
    if kind == "score":
        n, d, k = case["n"], case["d"], case["k"]
        return {"bytes": 4.0 * n * d + 8.0 * n + 24.0 * k * d * d,
                "flops": n * d * d + (3 * k + k * (k - 1) / 2) * d ** 3 / 3.0}
    if kind == "fit":
        n, d, k = case["n"], case["d"], case["k"]
        b, f = _gauss_sweep_work(n, d, k, False)
        return {"bytes": 8.0 * n * d + case["iters"] * b, "flops": case["iters"] * f}
    out = [_gauss_sweep_work(n, d, k, False) for n, d, k in _batch_shapes(case)]
    return {"bytes": sum(b for b, _ in out), "flops": sum(f for _, f in out)}


# ----------------------------------------------------------------------------- exact
def _mvlgamma(a, d):
    j = torch.arange(d, dtype=torch.float64)
    return torch.lgamma(a[:, None] - j[None, :] / 2).sum(1)


def _niw_lml(n, total, scatter, d):
    """Log marginal likelihood of NIW statistics (kappa = 1, m = 0, nu = d + 3, psi = I), in the
    parametrisation of the reference: the scale matrix is nu psi.  n, total, scatter: float64, batched."""
    k0, v0 = 1.0, d + 3.0
    kp, vp = k0 + n, v0 + n
    m = total / kp[:, None]
    psi = (v0 * torch.eye(d, dtype=torch.float64, device=scatter.device) + scatter
           - kp[:, None, None] * m[:, :, None] * m[:, None, :]) / vp[:, None, None]
    ld = torch.linalg.slogdet(psi)[1].cpu()
    n, kp, vp = n.cpu(), kp.cpu(), vp.cpu()
    v = (-n * d / 2 * math.log(math.pi) + _mvlgamma(vp / 2, d) - _mvlgamma(torch.full_like(vp, v0 / 2), d)
         + v0 / 2 * d * math.log(v0) - vp / 2 * (d * torch.log(vp) + ld) + d / 2 * torch.log(k0 / kp))
    return torch.where(n > 0, v, torch.zeros_like(v))


def exact(case, seed):
    if case["kind"] != "score":
        return None   # labels are draws; the other numbers follow from them
    n, d, K = case["n"], case["d"], case["k"]
    x, lab, sub = _score_inputs(case, seed)
    x = x.double()
    slot = torch.from_numpy(2 * (lab.astype(np.int64) - 1) + (sub - 1)).cuda()
    cnt = torch.bincount(slot, minlength=2 * K).double()
    tot = torch.zeros(2 * K, d, dtype=torch.float64, device="cuda").index_add_(0, slot, x)
    sc = torch.stack([x[slot == s].T @ x[slot == s] for s in range(2 * K)])
    cnt, tot, sc = cnt.view(K, 2), tot.view(K, 2, d), sc.view(K, 2, d, d)
    cnt = torch.cat([cnt.sum(1, keepdim=True), cnt], 1)
    tot = torch.cat([tot.sum(1, keepdim=True), tot], 1)
    sc = torch.cat([sc.sum(1, keepdim=True), sc], 1)
    lml = _niw_lml(cnt.reshape(-1), tot.reshape(-1, d), sc.reshape(-1, d, d), d).view(K, 3)
    c = cnt.cpu()
    split = (math.log(ALPHA) + torch.lgamma(c[:, 1]) + lml[:, 1] + torch.lgamma(c[:, 2]) + lml[:, 2]
             - (torch.lgamma(c[:, 0]) + lml[:, 0]))
    split[(c[:, 1] == 0) | (c[:, 2] == 0)] = math.nan
    merge = torch.full((K, K), math.nan, dtype=torch.float64)
    i, j = torch.triu_indices(K, K, 1)
    if i.numel():
        both = _niw_lml(cnt[i.cuda(), 0] + cnt[j.cuda(), 0], tot[i.cuda(), 0] + tot[j.cuda(), 0],
                        sc[i.cuda(), 0] + sc[j.cuda(), 0], d)
        ni, nj, a = c[i, 0], c[j, 0], ALPHA
        hr = (-math.log(a) + math.lgamma(a) - 2 * math.lgamma(0.5 * a) + torch.lgamma(ni + nj) - torch.lgamma(ni + nj + a)
              + torch.lgamma(ni + 0.5 * a) - torch.lgamma(ni) - torch.lgamma(nj) + torch.lgamma(nj + 0.5 * a)
              + both - lml[i, 0] - lml[j, 0])
        hr[(ni == 0) | (nj == 0)] = math.nan
        merge[i, j] = hr
    return dict(count=None, total=tot.cpu(), scatter=sc.cpu(), lml=lml, split=split, merge=merge)
