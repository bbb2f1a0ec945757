"""Workloads of the searchlight alignment library, as its users call it.

Every case is one pass through a public entry point: the device-resident plan
(``hyperalignment_b200.plan.Plan``) for programs that keep their data on the GPU, or the
reference-shaped wrapper (``hyperalignment_b200.hyperalignment_c``) for programs that call with
host arrays.  Shapes are those of the package's workload generators (``workloads.py``) and of
``bench.py``: vertices on a Fibonacci sphere, one searchlight per centre, subject time series
related by block-local rotations plus noise.

``prepare`` makes inputs and plan from the seed and the case's geometry, ``run`` is one pass, ``work`` counts the
bytes and operations a pass cannot do without, and ``exact`` gives the same outputs in plain
float64 torch and numpy.
"""

from __future__ import annotations

import math

import numpy as np
import torch

from hyperalignment_b200 import _lib as L
from hyperalignment_b200 import hyperalignment_c as H
from hyperalignment_b200 import workloads as W
from hyperalignment_b200.plan import Plan

SOLVERS = {"tc": L.SOLVER_TC, "mixed": L.SOLVER_MIXED, "fp32": L.SOLVER_FP32, "fp64": L.SOLVER_FP64}
N_FEAT = 65


# -------------------------------------------------------------------------------------------------
# cases
# -------------------------------------------------------------------------------------------------

def _case(path, nv, nt, lo, hi, count=0, **more):
    """nv vertices, nt time points, searchlights of lo..hi vertices around `count` evenly spaced
    centres (0: around every vertex)."""
    return {"path": path, "nv": nv, "nt": nt, "lo": lo, "hi": hi, "count": count, **more}


def listed():
    return [
        # the smallest call: a coarse sphere with tiny searchlights, where launches are the time
        {"name": "small_call", **_case("procrustes", 162, 40, 8, 24, solver="tc", reflection=True, scaling=False,
                                       csc=False, singular=0.0)},
        # the reference wrapper's call on host arrays, lists in and a dense matrix out (config 1 of bench.py)
        {"name": "wrapper_dense", **_case("dense", 2562, 200, 71, 78, reflection=True, scaling=False)},
        # one alignment of the hemisphere template loop, a tenth of the searchlights exactly singular
        # (the default workload of bench.py)
        {"name": "template_pair", **_case("procrustes", 10242, 400, 100, 300, solver="tc", reflection=True,
                                          scaling=True, csc=False, singular=0.1)},
        # the shapes of the reference's published run: long series, searchlights of about 121
        {"name": "long_series", **_case("procrustes", 9675, 1818, 90, 170, solver="tc", reflection=True,
                                        scaling=False, csc=True, singular=0.0)},
        # the widest searchlights the solvers take
        {"name": "wide_searchlights", **_case("procrustes", 2562, 1000, 301, 512, count=854, solver="tc",
                                              reflection=True, scaling=True, csc=False, singular=0.0)},
        # rotations only: det(T) > 0 is forced, with the global scale
        {"name": "no_reflection", **_case("procrustes", 2562, 200, 71, 78, solver="mixed", reflection=False,
                                          scaling=True, csc=True, singular=0.0)},
        # ridge at one penalty
        {"name": "ridge", **_case("ridge", 2562, 400, 100, 300, alpha=10.0, csc=True)},
        # cross-validated grid search over 10 penalties x 4 PC counts, float64
        {"name": "ridge_grid", **_case("grid", 10242, 500, 50, 500, count=512, bits=64, folds=5)},
        # learned proposal with the grid as its fallback, the mixed-precision form
        {"name": "learned_mixed", **_case("learned", 10242, 500, 50, 500, count=512, bits=32, folds=5)},
        # searchlight PCA template of a group, host arrays
        {"name": "pca_template", **_case("pca", 2562, 400, 100, 300, count=256, subjects=10)},
        # Procrustes template of a group, host arrays
        {"name": "procrustes_template", **_case("template", 2562, 300, 60, 200, subjects=4, scaling=True,
                                                zscore=True, level2=1)},
        # evaluation: correlation of aligned held-out data with a target
        {"name": "evaluation", **_case("correlation", 10242, 400, 100, 300)},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    path = rng.choice(["procrustes", "procrustes", "procrustes", "dense", "ridge", "grid", "learned", "pca",
                       "template", "correlation"])
    if path in ("procrustes", "dense", "template", "correlation"):
        nv = _log_int(rng, 162, 5000)
        hi = min(_log_int(rng, 20, 320), nv // 2)
        nt = max(_log_int(rng, 40, 1000), hi + hi // 4)
        lo = max(8, int(hi * rng.uniform(0.3, 1.0)))
        if path == "procrustes":
            refl = rng.random() < 0.8
            return _case(path, nv, nt, lo, hi, solver="tc" if refl else "mixed", reflection=refl,
                         scaling=rng.random() < 0.5, csc=rng.random() < 0.5,
                         singular=0.1 if refl and rng.random() < 0.25 else 0.0)
        if path == "dense":
            return _case(path, min(nv, 3000), nt, lo, hi, reflection=True, scaling=rng.random() < 0.5)
        if path == "template":
            return _case(path, min(nv, 2562), min(nt, 500), lo, min(hi, 200), subjects=rng.randint(2, 4),
                         scaling=rng.random() < 0.5, zscore=rng.random() < 0.7, level2=rng.randint(0, 1))
        return _case(path, nv, nt, lo, hi)
    hi = _log_int(rng, 50, 500 if path in ("grid", "learned") else 300)
    lo = max(20, int(hi * rng.uniform(0.2, 1.0)))
    if path == "ridge":
        return _case(path, 2562, _log_int(rng, 100, 500), lo, hi, count=_log_int(rng, 64, 2000),
                     alpha=10.0 ** rng.uniform(-1, 3), csc=rng.random() < 0.5)
    if path == "pca":
        nt = max(hi, rng.randint(120, 500))
        return _case(path, 2562, nt, lo, hi, count=rng.randint(16, 64), subjects=rng.randint(2, 10))
    return _case(path, 2562, rng.randint(300, 500), lo, hi, count=rng.randint(16, 48),
                 bits=64 if path == "grid" else rng.choice([32, 64]), folds=rng.randint(4, 6))


# -------------------------------------------------------------------------------------------------
# inputs
# -------------------------------------------------------------------------------------------------

def _sphere(n):
    return torch.from_numpy(W.fibonacci_sphere(n)).cuda()


def _searchlights(case):
    """k-nearest-neighbour searchlights: members ascending, geodesic distances to the centre.  The geometry
    is the case's (one cortical mesh), the data the seed's."""
    nv = case["nv"]
    pts = _sphere(nv)
    count = case["count"] or nv
    centres = (torch.arange(count, device="cuda") * nv) // count
    sizes = torch.from_numpy(np.random.default_rng(nv).integers(case["lo"], case["hi"] + 1, count)).cuda()
    kmax = int(sizes.max())
    dot = pts[centres] @ pts.T
    near = torch.topk(dot, kmax, dim=1).indices
    keep = torch.arange(kmax, device="cuda")[None, :] < sizes[:, None]
    near = torch.where(keep, near, nv).sort(dim=1).values  # ascending, the absent ones last
    keep = near < nv
    chord = (pts[near.clamp(max=nv - 1)] - pts[centres][:, None, :]).norm(dim=2)
    dist = (2.0 * torch.asin((0.5 * chord).clamp(max=1.0)))[keep]
    offsets = torch.zeros(count + 1, dtype=torch.int64, device="cuda")
    offsets[1:] = sizes.cumsum(0)
    d = dist.cpu().numpy()
    return W.Searchlights(near[keep].to(torch.int32).cpu().numpy(), offsets.to(torch.int32).cpu().numpy(), d,
                          1.0001 * float(d.max()), nv)


def _normal(gen, *shape):
    return torch.randn(*shape, generator=gen, device="cuda", dtype=torch.float64)


def _rotate(X, cells, members, gen):
    """X (nv x nt, a vertex a row) with an orthogonal map of its own in every cell."""
    n_cells, width = members.shape
    g = _normal(gen, n_cells, width, width)
    real = members >= 0
    both = real[:, :, None] & real[:, None, :]
    g = torch.where(both, g, torch.eye(width, device="cuda", dtype=torch.float64)[None] * (~real)[:, :, None])
    q, r = torch.linalg.qr(g)
    q = q * torch.sign(torch.diagonal(r, dim1=1, dim2=2))[:, None, :]
    out = torch.bmm(q.transpose(1, 2), X[members.clamp(min=0)] * real[:, :, None])
    Y = torch.empty_like(X)
    Y[members[real]] = out[real]
    return Y


def _subjects(case, gen, n, noise=0.2, ar=0.0, span=1.0):
    """n subjects as nv x nt float64 CUDA tensors (column-major nt x nv): a shared latent series, a
    block-local rotation and noise per subject."""
    nv, nt = case["nv"], case["nt"]
    pts = _sphere(nv)
    owner = (pts @ _sphere(max(1, nv // 64)).T).argmax(dim=1)
    order = torch.argsort(owner, stable=True)
    per = torch.bincount(owner)
    per = per[per > 0]
    start = per.cumsum(0) - per
    k = torch.arange(int(per.max()), device="cuda")
    members = torch.where(k[None, :] < per[:, None], order[(start[:, None] + k[None, :]).clamp(max=nv - 1)], -1)
    latent = _normal(gen, nv, nt)
    amp = noise * span ** ((pts[:, 2:3] + 1.0) / 2.0)
    out = []
    for _ in range(n):
        e = _normal(gen, nt, nv)
        if ar:
            c = math.sqrt(1.0 - ar * ar)
            for t in range(1, nt):
                e[t].mul_(c).add_(e[t - 1], alpha=ar)
        out.append((_rotate(latent, owner, members, gen) + amp * e.T).contiguous())
    return out


def _duplicate_columns(X, sls, frac, seed):
    """X (nt x nv) with columns copied until about frac of the searchlights are exactly singular."""
    Xh = X.T.cpu().numpy().copy()
    W.duplicate_columns_to_fraction(Xh, sls, frac, np.random.default_rng(seed))
    return torch.from_numpy(np.ascontiguousarray(Xh.T)).cuda()


def _splits(case, n_rows, seed):
    return H.ensemble_indices(n_rows, 1, case["folds"], 10, 10, seed)


def _proposal(gen):
    """A perceptron whose proposals are confident for most searchlights."""
    C = len(W.GRID_ALPHAS) * len(W.GRID_NPCS)
    parts = []
    for n_in, n_out, gain in ((N_FEAT, 128, 1.0), (128, 128, 1.0), (128, C, 60.0)):
        a = 1.0 / math.sqrt(n_in)
        for rows, g in ((n_in, gain), (1, gain)):
            u = torch.rand(rows, n_out, generator=gen, device="cuda")
            parts.append(((2.0 * u - 1.0) * a * g).reshape(-1))
    return torch.cat(parts).float().contiguous()


def _inputs(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    sls = _searchlights(case)
    path = case["path"]
    s = {"case": case, "sls": sls}
    if path in ("pca", "template"):
        s["dms"] = _subjects(case, gen, case["subjects"])
        return s
    if path in ("grid", "learned"):
        s["Y"], s["X"] = _subjects(case, gen, 2, ar=0.5, span=30.0)
        n_fit = case["nt"] if path == "grid" else (case["nt"] * 4) // 5
        s["rows"] = np.arange(n_fit, dtype=np.int32)
        s["train"], s["test"] = _splits(case, n_fit, seed)
        if path == "learned":
            s["params"] = _proposal(gen)
        return s
    s["Y"], s["X"] = _subjects(case, gen, 2)
    if case.get("singular"):
        s["X"] = _duplicate_columns(s["X"], sls, case["singular"], seed)
    if path == "correlation":
        s["gen"] = gen
    return s


def _host(t):
    """nv x nt CUDA tensor -> nt x nv Fortran-order array."""
    return t.cpu().numpy().T


def prepare(case, seed):
    s = _inputs(case, seed)
    sls, path = s["sls"], case["path"]
    if path == "dense":
        s["X"], s["Y"] = _host(s["X"]), _host(s["Y"])
        s["lists"] = sls.as_lists()
        return s
    if path in ("pca", "template"):
        s["dms"] = [_host(d) for d in s["dms"]]
        s["lists"] = sls.as_lists()
        return s
    plan = Plan(case["nt"], case["nv"], sls.indices, sls.offsets, sls.dists, sls.radius)
    s["plan"] = plan
    s["values"] = torch.zeros(plan.nnz, dtype=torch.float64, device="cuda")
    if path == "grid":
        plan.set_grid_precision(case["bits"])
        grid = len(W.GRID_ALPHAS) * len(W.GRID_NPCS)
        s["best"] = torch.zeros(plan.count, dtype=torch.int32, device="cuda")
        s["cost"] = torch.zeros(plan.count, grid, dtype=torch.float64, device="cuda")
    elif path == "learned":
        plan.set_grid_precision(case["bits"])
        s["choice"] = torch.zeros(plan.count, dtype=torch.int32, device="cuda")
        s["prob"] = torch.zeros(plan.count, dtype=torch.float32, device="cuda")
    elif path == "correlation":
        s["values"] = _normal(s.pop("gen"), plan.nnz) / math.sqrt(0.5 * (case["lo"] + case["hi"]))
        s["r"] = torch.zeros(case["nv"], dtype=torch.float64, device="cuda")
        s["aligned"] = torch.zeros(case["nv"], case["nt"], dtype=torch.float64, device="cuda")
    return s


# -------------------------------------------------------------------------------------------------
# one pass
# -------------------------------------------------------------------------------------------------

def run(s):
    case = s["case"]
    path = case["path"]
    if path == "dense":
        sls, dists = s["lists"]
        return H.searchlight_procrustes(s["X"], s["Y"], sls, dists, s["sls"].radius, backend="b200",
                                        reflection=case["reflection"], scaling=case["scaling"], n_jobs=8)
    if path == "template":
        sls, dists = s["lists"]
        return H.searchlight_template(s["dms"], sls, dists, s["sls"].radius, reflection=True, scaling=case["scaling"],
                                      zscore_common=case["zscore"], level2_iter=case["level2"])
    if path == "pca":
        sls, dists = s["lists"]
        return H.searchlight_pca_template(s["dms"], sls, dists, s["sls"].radius)
    plan, values = s["plan"], s["values"]
    X, Y = s["X"].data_ptr(), s["Y"].data_ptr()
    stream = torch.cuda.current_stream().cuda_stream
    if path == "correlation":
        plan.aligned_correlation_device(X, Y, values.data_ptr(), s["r"].data_ptr(), s["aligned"].data_ptr(),
                                        stream=stream)
        return s["r"], s["aligned"]
    values.zero_()  # the calls accumulate
    if path == "procrustes":
        plan.procrustes_device(X, Y, values.data_ptr(), reflection=case["reflection"], scaling=case["scaling"],
                               solver=SOLVERS[case["solver"]], out_kind=L.OUT_CSC if case["csc"] else L.OUT_CSR,
                               stream=stream)
        return values
    if path == "ridge":
        plan.ridge_device(X, Y, values.data_ptr(), case["alpha"], out_kind=L.OUT_CSC if case["csc"] else L.OUT_CSR,
                          stream=stream)
        return values
    if path == "grid":
        plan.ridge_grid_device(X, Y, values.data_ptr(), s["best"].data_ptr(), W.GRID_ALPHAS, W.GRID_NPCS, s["train"],
                               s["test"], d_cost=s["cost"].data_ptr(), stream=stream)
        return values, s["best"], s["cost"]
    plan.ridge_learned_device(X, Y, s["rows"], W.GRID_ALPHAS, W.GRID_NPCS, s["params"].data_ptr(), 0.6, s["train"],
                              s["test"], values.data_ptr(), s["choice"].data_ptr(), s["prob"].data_ptr(),
                              stream=stream)
    return values, s["choice"], s["prob"]


# -------------------------------------------------------------------------------------------------
# what a pass cannot do without
# -------------------------------------------------------------------------------------------------

def _moments(case):
    """Searchlights and the means of n, n^2 and n^3 for sizes uniform in lo..hi."""
    n = np.arange(case["lo"], case["hi"] + 1, dtype=np.float64)
    return case["count"] or case["nv"], n.mean(), (n * n).mean(), (n ** 3).mean()


def work(case):
    """Inputs once, outputs once; the operations of the reference's algorithm per searchlight: products
    over the time points, a decomposition of n x n (21 n^3 with both singular bases, 9 n^3 for a
    symmetric one), a product of its bases."""
    count, n1, n2, n3 = _moments(case)
    nv, nt, path = case["nv"], case["nt"], case["path"]
    # stored entries of the pattern: a vertex meets those within two searchlight radii of its own
    nnz = min(float(nv) * nv, nv * 4.0 * n1 if not case["count"] else count * n2)
    io = 2.0 * 8 * nv * nt + 8.0 * nnz
    solve = 2.0 * nt * n2 + 23.0 * n3
    if path == "procrustes":
        return {"bytes": io, "flops": count * solve}
    if path == "dense":
        return {"bytes": 2.0 * 8 * nv * nt + 8.0 * nv * nv, "flops": count * solve}
    if path == "template":
        solves = case["subjects"] - 1 + case["level2"] * case["subjects"]
        return {"bytes": 8.0 * nv * nt * (case["subjects"] + 1),
                "flops": solves * (count * solve + 2.0 * nt * nnz)}
    if path == "pca":
        return {"bytes": 8.0 * nv * nt * (case["subjects"] + 1),
                "flops": count * (2.0 * case["subjects"] * n1 * nt * min(nt, case["subjects"] * n1)
                                  + 9.0 * min(nt, case["subjects"] * n1) ** 3 + 4.0 * nt * n2 + 23.0 * n3)}
    if path == "correlation":
        return {"bytes": 8.0 * nnz + 3.0 * 8 * nv * nt, "flops": 2.0 * nt * nnz}
    if path == "ridge":
        return {"bytes": io, "flops": count * (4.0 * nt * n2 + n3 / 3.0 + 2.0 * n3)}
    # per model: two products over its training rows, the decomposition, the test predictions of every penalty
    tested = nt / float(case["folds"])
    model = 4.0 * nt * n2 + 9.0 * n3 + 2.0 * n3 + 2.0 * len(W.GRID_ALPHAS) * tested * n2
    if path == "grid":
        return {"bytes": io, "flops": count * case["folds"] * model}
    return {"bytes": io, "flops": count * (4.0 * nt * n2 + 9.0 * n3 + 4.0 * n3)}


# -------------------------------------------------------------------------------------------------
# the same outputs in plain float64
# -------------------------------------------------------------------------------------------------

def _padded(sls):
    """Members of every searchlight, padded with -1 to the widest."""
    sizes = np.diff(sls.offsets)
    m = np.full((sls.count, int(sizes.max())), -1, dtype=np.int64)
    m[np.arange(m.shape[1])[None, :] < sizes[:, None]] = sls.indices
    return torch.from_numpy(m).cuda()


def _weights(sls):
    w = (sls.radius - torch.from_numpy(sls.dists).cuda()) / sls.radius
    idx = torch.from_numpy(sls.indices.astype(np.int64)).cuda()
    total = torch.zeros(sls.nv, dtype=torch.float64, device="cuda").index_add_(0, idx, w)
    flat = w / total[idx]
    m = _padded(sls)
    out = torch.zeros(m.shape, dtype=torch.float64, device="cuda")
    out[m >= 0] = flat
    return out


def _polar(A):
    """Polar factors of a batch by the scaled cubic iteration, with their nuclear norms."""
    norm = torch.linalg.matrix_norm(A)[:, None, None]
    Z = A / norm
    low = 1e-9
    for _ in range(45):
        a = min(math.sqrt(3.0 / (1.0 + low + low * low)), 1.65)
        a = 1.0 if a < 1.01 else a
        low = min(1.0, 0.5 * a * low * (3.0 - a * a * low * low))
        Z = 1.5 * a * Z - (0.5 * a ** 3) * torch.bmm(Z, torch.bmm(Z.transpose(1, 2), Z))
    return Z, (Z * A).sum(dim=(1, 2))


def _rotation(A, real):
    """The same without reflections, by SVD (csrc/ha_searchlight.c:593-656 of the reference)."""
    T, total = torch.zeros_like(A), torch.zeros(A.shape[0], dtype=torch.float64, device=A.device)
    for i in range(A.shape[0]):
        n = int(real[i].sum())
        u, s, vt = np.linalg.svd(A[i, :n, :n].cpu().numpy())
        t = u @ vt
        if np.linalg.slogdet(t)[0] < 0:
            t -= 2.0 * np.outer(u[:, -1], vt[-1])
            s[-1] = -s[-1]
        T[i, :n, :n] = torch.from_numpy(t).cuda()
        total[i] = float(s.sum())
    return T, total


def _scatter(sls, blocks, scale=None):
    """Dense nv x nv sum of the weighted local results; blocks(members, real) of a batch."""
    nv = sls.nv
    members, w = _padded(sls), _weights(sls)
    D = torch.zeros(nv * nv, dtype=torch.float64, device="cuda")
    step = max(1, int(4e7) // members.shape[1] ** 2)
    for b in range(0, members.shape[0], step):
        m = members[b:b + step]
        real = m >= 0
        T = blocks(b, m.clamp(min=0), real) * w[b:b + step][:, :, None]
        at = m[:, :, None] * nv + m[:, None, :]
        both = real[:, :, None] & real[:, None, :]
        D.index_add_(0, at[both], T[both])
    return D.view(nv, nv)


def _procrustes(X, Y, sls, reflection, scaling):
    """Dense W of the searchlight Procrustes alignment of X onto Y (nv x nt)."""
    nt = X.shape[1]
    var = X.var(dim=1, unbiased=False)

    def blocks(_, m, real):
        both = real[:, :, None] & real[:, None, :]
        A = torch.bmm(X[m], Y[m].transpose(1, 2)) * both
        if reflection:
            # an identity block in the padding keeps it apart
            fill = torch.diag_embed((~real).to(torch.float64))
            top = torch.linalg.matrix_norm(A)[:, None, None] / math.sqrt(A.shape[1])
            T, total = _polar(A + fill * top)
            total = total - (~real).sum(dim=1) * top[:, 0, 0]
        else:
            T, total = _rotation(A, real)
        if scaling:
            T = T * (total / ((var[m] * real).sum(dim=1) * nt))[:, None, None]
        return T * both

    return _scatter(sls, blocks)


def _entries(D, sls, csc):
    """The stored entries of D over the union pattern of the searchlights, in column or row order."""
    members = _padded(sls)
    M = torch.zeros(sls.count, sls.nv + 1, dtype=torch.float32, device="cuda")
    M.scatter_(1, torch.where(members >= 0, members, sls.nv), 1.0)
    M = M[:, :-1]
    return (D.T if csc else D)[(M.T @ M) > 0]


def _zscore(A):
    m = A.mean(dim=1, keepdim=True)
    v = (A * A).mean(dim=1, keepdim=True) - m * m
    return torch.where(v < 1e-30, torch.zeros_like(A), (A - m) / v.clamp(min=1e-300).sqrt())


def _template(case, s):
    dms, sls = s["dms"], s["sls"]
    z = _zscore if case["zscore"] else (lambda a: a)

    def align(d, target):
        return _procrustes(d, target, sls, True, case["scaling"]).T @ d

    common, aligned = dms[0], [dms[0]]
    for d in dms[1:]:
        aligned.append(z(align(d, common)))
        common = z((common + aligned[-1]) / 2)
    for _ in range(case["level2"]):
        total = sum(aligned)
        for k, d in enumerate(dms):
            aligned[k] = align(d, z((total - aligned[k]) / (len(dms) - 1)))
    total = sum(aligned)
    return (_zscore(total) if case["zscore"] else total / len(dms)).T.contiguous()


def _pca(case, s):
    sls, dms = s["sls"], [d.cpu().numpy() for d in s["dms"]]
    ns, members, w = len(dms), _padded(sls).cpu().numpy(), _weights(sls).cpu().numpy()
    out = np.zeros((case["nt"], case["nv"]))
    for i in range(sls.count):
        m = members[i][members[i] >= 0]
        n = m.size
        X = np.concatenate([d[m] for d in dms]).T
        G = X @ X.T if X.shape[0] <= X.shape[1] else X.T @ X
        lam, vec = np.linalg.eigh(G)
        vec, lam = vec[:, ::-1][:, :n], np.maximum(lam[::-1][:n], 0.0)
        tmpl = (vec * np.sqrt(lam) if X.shape[0] <= X.shape[1] else X @ vec) / math.sqrt(ns)
        u, _, vt = np.linalg.svd(tmpl.T @ sum(d[m].T for d in dms))
        out[:, m] += (tmpl @ (u @ vt)) * w[i, :n]
    return out


def _fit(X, Y, alphas, npcs):
    """Betas over the grid of one training block: a list over PC counts per penalty."""
    u, s, vt = np.linalg.svd(X, full_matrices=False)
    q = u.T @ Y
    grid = []
    for a in alphas:
        beta, row = np.zeros((X.shape[1], Y.shape[1])), []
        for p, hi in enumerate(npcs):
            lo = npcs[p - 1] if p else 0
            k = slice(min(lo, s.size), min(hi, s.size))
            beta = beta + (vt[k].T * (s[k] / (a + s[k] ** 2))) @ q[k]
            row.append(beta)
        grid.append(row)
    return grid


def _grid(case, s):
    X, Y, sls = _host(s["X"]), _host(s["Y"]), s["sls"]
    alphas, npcs = [float(a) for a in W.GRID_ALPHAS], [int(p) for p in W.GRID_NPCS]
    members = _padded(sls).cpu().numpy()
    tested = np.zeros(case["nt"])
    for t in s["test"]:
        tested[t] += 1
    betas = torch.zeros(sls.count, members.shape[1], members.shape[1], dtype=torch.float64)
    best, cost = [], []
    for i in range(sls.count):
        m = members[i][members[i] >= 0]
        models = [_fit(X[np.ix_(tr, m)], Y[np.ix_(tr, m)], alphas, npcs) for tr in s["train"]]
        c = np.zeros((len(alphas), len(npcs)))
        for a in range(len(alphas)):
            for p in range(len(npcs)):
                pred = np.zeros((case["nt"], m.size))
                for model, te in zip(models, s["test"]):
                    pred[te] += X[np.ix_(te, m)] @ model[a][p] / tested[te][:, None]
                c[a, p] = ((Y[:, m] - pred) ** 2).sum()
        g = int(c.argmin())
        a, p = divmod(g, len(npcs))
        best.append(g)
        cost.append(c.reshape(-1))
        betas[i, :m.size, :m.size] = torch.from_numpy(sum(model[a][p] for model in models) / len(models))
    betas = betas.cuda()
    D = _scatter(sls, lambda b, m, real: betas[b:b + m.shape[0]])
    return _entries(D, sls, True), torch.tensor(best, dtype=torch.int32), torch.from_numpy(np.array(cost))


def exact(case, seed):
    path = case["path"]
    count, _, _, n3 = _moments(case)
    if case.get("singular") or path == "learned":
        return None  # a null space has no one completion; the proposal's precision decides its choices
    if path == "grid" and count * case["folds"] * n3 > 48 * 5 * 2e7:
        return None  # a minute and more of host SVDs
    s = _inputs(case, seed)
    sls = s["sls"]
    if path == "pca":
        return _pca(case, s)
    if path == "template":
        return _template(case, s)
    if path == "grid":
        return _grid(case, s)
    X, Y = s["X"], s["Y"]
    if path == "dense":
        return _procrustes(X, Y, sls, case["reflection"], case["scaling"])
    if path == "procrustes":
        return _entries(_procrustes(X, Y, sls, case["reflection"], case["scaling"]), sls, case["csc"])
    if path == "ridge":
        def blocks(_, m, real):
            both = real[:, :, None] & real[:, None, :]
            Xs, Ys = X[m] * real[:, :, None], Y[m] * real[:, :, None]
            G = torch.bmm(Xs, Xs.transpose(1, 2)) + case["alpha"] * torch.eye(m.shape[1], device="cuda",
                                                                              dtype=torch.float64)
            return torch.cholesky_solve(torch.bmm(Xs, Ys.transpose(1, 2)), torch.linalg.cholesky(G)) * both
        return _entries(_scatter(sls, blocks), sls, case["csc"])
    # correlation: the same values over the union pattern
    D = torch.zeros(case["nv"], case["nv"], dtype=torch.float64, device="cuda")
    pattern = _entries(torch.arange(case["nv"] ** 2, device="cuda").view(case["nv"], case["nv"]), sls, True)
    D.view(-1)[pattern] = _normal(s["gen"], pattern.numel()) / math.sqrt(0.5 * (case["lo"] + case["hi"]))
    aligned = D.T @ X
    return (_zscore(aligned) * _zscore(Y)).mean(dim=1), aligned
