"""The blocked kernels at the edges of their tiles, against the CPU oracle."""

import numpy as np
import pytest

from hyperalignment_b200 import _lib as L
from hyperalignment_b200.plan import Plan
from oracle import ha_oracle as O

pytestmark = pytest.mark.gpu


def one_each(sizes, nt, seed):
    """Gaussian series and one searchlight of every size over a common vertex set."""
    rng = np.random.default_rng(seed)
    nv = max(sizes)
    X, Y = rng.standard_normal((nt, nv)), rng.standard_normal((nt, nv))
    idx = np.concatenate([np.sort(rng.choice(nv, n, replace=False)) for n in sizes]).astype(np.int32)
    off = np.concatenate([[0], np.cumsum(sizes)]).astype(np.int32)
    return X, Y, idx, off


def upload(X):
    import torch
    return torch.from_numpy(np.asfortranarray(X).ravel(order="F")).cuda()


# A Gaussian X of 700 samples has cond(X^T X) < 200 for n <= 512, so normal equations solved in
# float64 carry at most about 200 * 512 * 2.2e-16 = 2e-11; four times that is allowed.
@pytest.mark.parametrize("csc", [False, True])
def test_ridge_tile_edges(gpu, csc):
    import torch
    sizes = [1, 2, 31, 63, 64, 65, 127, 128, 129, 200, 255, 257, 511, 512]
    X, Y, idx, off = one_each(sizes, 700, 3)
    dX, dY = upload(X), upload(Y)
    for s, n in enumerate(sizes):
        sl = idx[off[s]:off[s + 1]]
        plan = Plan(700, X.shape[1], sl, np.array([0, n]), weights=np.ones(n))
        vals = torch.zeros(plan.nnz, dtype=torch.float64, device="cuda")
        plan.ridge_device(dX.data_ptr(), dY.data_ptr(), vals.data_ptr(), 0.5,
                          out_kind=L.OUT_CSC if csc else L.OUT_CSR)
        got = vals.cpu().numpy().reshape(n, n)
        plan.close()
        ref = O.ridge(X[:, sl], Y[:, sl], 0.5)
        err = np.linalg.norm((got.T if csc else got) - ref) / np.linalg.norm(ref)
        assert err <= 8e-11, (n, err)


def test_ridge_without_penalty_on_singular_data_writes_zeros(gpu):
    import torch
    rng = np.random.default_rng(4)
    X, Y = rng.standard_normal((300, 130)), rng.standard_normal((300, 130))
    X[:, 100] = 0.0
    dX, dY = upload(X), upload(Y)
    plan = Plan(300, 130, np.arange(130), np.array([0, 130]), weights=np.ones(130))
    vals = torch.zeros(plan.nnz, dtype=torch.float64, device="cuda")
    plan.ridge_device(dX.data_ptr(), dY.data_ptr(), vals.data_ptr(), 0.0)
    assert plan.stats()["n_unconverged"] == 1
    assert not vals.any()
    plan.close()


# R is rounded to float32 (6e-8 relative per element); everything else is float64.
@pytest.mark.parametrize("nt,ns,sizes", [
    (64, 3, [1, 2, 31, 63, 64]),          # Gram order nt: a whole tile; also ns n < nt (vertex side)
    (65, 2, [1, 16, 32, 33, 64, 65]),     # one row more than a tile
    (130, 3, [5, 43, 44, 64, 65, 128]),
    (400, 1, [63, 129, 257]),             # vertex side only
])
def test_pca_template_tile_edges(gpu, nt, ns, sizes):
    from hyperalignment_b200 import hyperalignment_c as H
    rng = np.random.default_rng(nt)
    X, _, idx, off = one_each(sizes, nt, nt)
    dms = [X @ np.linalg.qr(rng.standard_normal((X.shape[1],) * 2))[0] + 0.1 * rng.standard_normal(X.shape)
           for _ in range(ns)]
    sls = [idx[off[s]:off[s + 1]] for s in range(len(sizes))]
    got = H.searchlight_pca_template(dms, sls, None, 1.0)
    ref = O.searchlight_pca_template(dms, idx, off, None, 1.0)
    assert np.linalg.norm(got - ref) / np.linalg.norm(ref) <= 1e-6


# Costs are sums of squares whose predictions carry the conditioning of G + alpha I (here < 1e4 for
# alpha >= 1e-1) times n eps; the repository's own bound for this search is 1e-8.
@pytest.mark.parametrize("nt,sizes,folds", [
    (150, [1, 2, 15, 16, 17, 63, 64, 65], 3),      # Gram and kernel forms of every model
    (300, [40, 127, 128, 129, 191, 193, 300], 4),  # both sides of the distinct-row count
])
def test_ridge_grid_tile_edges(gpu, nt, sizes, folds):
    from hyperalignment_b200 import hyperalignment_c as H
    rng = np.random.default_rng(nt)
    X, Y, idx, off = one_each(sizes, nt, nt)
    Y = 0.3 * X + Y
    tr = [rng.integers(0, nt, nt).astype(np.int32) for _ in range(folds)]
    te = [np.setdiff1d(np.arange(nt), t).astype(np.int32)[:65 + 3 * k] for k, t in enumerate(tr)]
    te[0] = te[0][:0]  # a model that tests nothing
    sls = [idx[off[s]:off[s + 1]] for s in range(len(sizes))]
    indptr, indices = H.sparse_pattern(sls, X.shape[1])
    data = np.zeros(indices.size)
    alphas, npcs = np.array([0.1, 3.0, 100.0]), [7, 16, 3, 33, 600]
    best, costs = H.searchlight_ridge_grid(X, Y, sls, indptr, indices, data, alphas, npcs, tr, te, return_costs=True)
    ref, rbest, rcosts = O.searchlight_ridge_grid_csc(X, Y, idx, off, indptr, indices, np.zeros(indices.size), alphas,
                                                      npcs, tr, te, None)
    np.testing.assert_allclose(costs, rcosts, rtol=1e-8, atol=0)
    np.testing.assert_array_equal(best, rbest)
    assert np.linalg.norm(data - ref) <= 1e-8 * np.linalg.norm(ref)


# lambda is accurate to n eps lambda_max: a singular value at relative s to 512 * 2.2e-16 / (2 s), and a
# Gaussian X of 700 rows keeps s > 0.1; the features are float32 (6e-8).
def test_features_at_eigen_solver_orders(gpu):
    import torch
    sizes = [1, 2, 3, 15, 16, 17, 18, 63, 64, 65, 128, 129, 192, 193, 256, 257, 384, 385, 511, 512]
    X, _, idx, off = one_each(sizes, 700, 9)
    plan = Plan(700, X.shape[1], idx, off, weights=np.ones(idx.size))
    f = torch.zeros((len(sizes), 65), dtype=torch.float32, device="cuda")
    dX = upload(X)
    plan.ridge_features_device(dX.data_ptr(), np.arange(700), f.data_ptr())
    got = f.cpu().numpy()
    plan.close()
    ref = O.ridge_features(X, idx, off, np.arange(700))
    np.testing.assert_allclose(got, ref, rtol=0, atol=2.5e-7)


_RESIDENT_SCRIPT = r"""
import sys
import numpy as np
import torch
sys.path.insert(0, sys.argv[1])
from hyperalignment_b200 import _lib as L
from hyperalignment_b200.plan import Plan
rng = np.random.default_rng(5)
sizes = [1, 15, 16, 17, 32, 33, 63, 64, 65, 80, 112, 127, 128, 129, 144, 145, 160, 176, 200, 208, 240, 241, 255, 256, 257, 300]
nv, nt = 300, 400
X = rng.standard_normal((nt, nv))
Y = X @ np.linalg.qr(rng.standard_normal((nv, nv)))[0] + 0.1 * rng.standard_normal((nt, nv))
X[:, 7] = X[:, 3]  # exactly singular searchlights among them
idx = np.concatenate([np.arange(n) for n in sizes]).astype(np.int32)
off = np.concatenate([[0], np.cumsum(sizes)]).astype(np.int32)
plan = Plan(nt, nv, idx, off, weights=np.ones(idx.size))
dX = torch.from_numpy(np.asfortranarray(X).ravel(order="F")).cuda()
dY = torch.from_numpy(np.asfortranarray(Y).ravel(order="F")).cuda()
out = {}
for kind in (L.OUT_CSR, L.OUT_CSC):
    v = torch.zeros(plan.nnz, dtype=torch.float64, device="cuda")
    for _ in range(2):
        v.zero_()
        plan.procrustes_device(dX.data_ptr(), dY.data_ptr(), v.data_ptr(), True, True, L.SOLVER_TC, kind)
    torch.cuda.synchronize()
    out[f"v{kind}"] = v.cpu().numpy()
    st = plan.searchlight_stats(0, len(sizes))
    out[f"s{kind}"], out[f"f{kind}"], out[f"u{kind}"] = st["sweeps"], st["flags"], st["s_max"]
    for s, T in enumerate(plan.local_transforms(0, len(sizes))):
        out[f"T{kind}_{s}"] = T
np.savez(sys.argv[2], **out)
"""


def test_resident_iteration_bitwise_equal(gpu, tmp_path):
    """The iteration on resident planes (one CTA up to 128, a pair up to 256) and the per-phase kernels
    (HA_B200_TC_RESIDENT=0) take the same products in the same order: transforms, values, iteration
    counts and flags are identical bit for bit, at and around every tile size."""
    import os
    import subprocess
    import sys
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    res = []
    for v in "01":
        path = tmp_path / f"r{v}.npz"
        subprocess.run([sys.executable, "-c", _RESIDENT_SCRIPT, root, str(path)],
                       env=dict(os.environ, HA_B200_TC_RESIDENT=v), check=True, timeout=300)
        res.append(np.load(path))
    for k in res[0].files:
        assert res[0][k].tobytes() == res[1][k].tobytes(), k


# The three-part split is exact to 2^-24 and the FP32 accumulator takes 6 nt / 16 additions: for nt <= 260
# a relative error of 2^-24 sqrt(6 * 260 / 16) * O(1) in the 2-norm, 5e-6 with a factor of eight to spare.
@pytest.mark.parametrize("nt", [1, 31, 32, 33, 65, 260])
def test_cross_covariance_tile_edges(gpu, hlib, nt):
    """Both size classes, one and two row tiles per block, one and two row blocks, short last stages."""
    rng = np.random.default_rng(nt)
    fp = L.c_float_p
    for n in [1, 2, 16, 17, 63, 80, 96, 97, 127, 128, 129, 144, 192, 193, 255, 256, 257, 288, 384, 385, 496, 512]:
        A = rng.standard_normal((n, nt)).astype(np.float32)
        B = rng.standard_normal((n, nt)).astype(np.float32)
        out = np.zeros((n, n), dtype=np.float32)
        assert hlib.ha_b200_tc_selftest(2, n, nt, A.ctypes.data_as(fp), B.ctypes.data_as(fp), out.ctypes.data_as(fp)) == 0
        ref = A.astype(np.float64) @ B.astype(np.float64).T
        # a product of few samples can cancel: bounded against the factors instead of the result
        scale = np.linalg.norm(A, axis=1)[:, None] * np.linalg.norm(B, axis=1)[None, :]
        assert (np.abs(out - ref) <= 5e-6 * scale).all(), n


def test_wide_iteration_bitwise_equal(gpu, tmp_path):
    """The 256-row tiles of the iteration past 256 vertices against the 128-row kernels: identical bits where
    the second row block and the column halves are one step wide, odd, or full, and K ends in half a stage."""
    import os
    import subprocess
    import sys
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    script = _RESIDENT_SCRIPT.replace(
        _RESIDENT_SCRIPT[_RESIDENT_SCRIPT.index("sizes = "):_RESIDENT_SCRIPT.index("X = rng")],
        "sizes = [200, 257, 271, 272, 273, 288, 320, 351, 384, 385, 400, 449, 496, 511, 512]\nnv, nt = 512, 600\n")
    res = []
    for v in "01":
        path = tmp_path / f"w{v}.npz"
        subprocess.run([sys.executable, "-c", script, root, str(path)],
                       env=dict(os.environ, HA_B200_TC_RESIDENT=v), check=True, timeout=300)
        res.append(np.load(path))
    for k in res[0].files:
        assert res[0][k].tobytes() == res[1][k].tobytes(), k


@pytest.mark.parametrize("nv,nt", [(1, 2), (15, 127), (16, 128), (17, 129), (33, 257), (162, 40)])
def test_template_column_edges(gpu, nv, nt):
    """Column statistics and the product with the transform at the edges of their tiles (16 columns, 128
    samples; four entries, 384 samples): the template against the oracle, which sums in the same order.  The
    transforms come from FP32 products of well-conditioned Gaussian series: 1e-5 of the template's norm."""
    from hyperalignment_b200 import hyperalignment_c as H
    rng = np.random.default_rng(100 * nv + nt)
    base = rng.standard_normal((nt, nv))
    dms = [base + 0.5 * rng.standard_normal((nt, nv)) for _ in range(2)]
    n = min(nv, max(1, nt // 4), 12)
    sls = [np.sort((c + np.arange(n)) % nv).astype(np.int32) for c in range(nv)]
    dists = [np.linspace(0.0, 0.5, n) for _ in range(nv)]
    idx, off = np.concatenate(sls), np.concatenate([[0], np.cumsum([n] * nv)]).astype(np.int32)
    out = H.searchlight_template(dms, sls, dists, 1.0, True, True, True, 1)
    ref = O.searchlight_template(dms, idx, off, np.concatenate(dists), 1.0, True, True, True, 1)
    assert np.linalg.norm(out - ref) <= 1e-5 * np.linalg.norm(ref)
