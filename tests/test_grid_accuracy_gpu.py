"""The float64 grid search, its eigen solver and the learned form's fit on data that is hard for them,
against the CPU oracle (LAPACK's SVD of the training rows)."""

import numpy as np
import pytest

from hyperalignment_b200.plan import Plan
from oracle import ha_oracle as O

pytestmark = pytest.mark.gpu


def upload(X):
    import torch
    return torch.from_numpy(np.asfortranarray(X).ravel(order="F")).cuda()


def test_eigen_solver_repeats_bit_for_bit(gpu):
    """1,500 matrices of order 2-96 at once, a warp each: the lanes of a warp share the tridiagonal matrix in
    shared memory while one of them rewrites it, so every run has to give the same bits whatever the lanes'
    pace.  lambda is accurate to n eps lambda_max and the features are float32 (6e-8)."""
    import torch
    rng = np.random.default_rng(11)
    nv, nt = 300, 140
    X = rng.standard_normal((nt, nv))
    sizes = rng.integers(2, 97, 1500)
    idx = np.concatenate([np.sort(rng.choice(nv, n, replace=False)) for n in sizes]).astype(np.int32)
    off = np.concatenate([[0], np.cumsum(sizes)]).astype(np.int32)
    plan = Plan(nt, nv, idx, off, weights=np.ones(idx.size))
    dX = upload(X)
    runs = []
    for _ in range(5):
        f = torch.zeros((sizes.size, 65), dtype=torch.float32, device="cuda")
        plan.ridge_features_device(dX.data_ptr(), np.arange(nt), f.data_ptr())
        runs.append(f.cpu().numpy())
    plan.close()
    for r in runs[1:]:
        assert r.tobytes() == runs[0].tobytes()
    np.testing.assert_allclose(runs[0], O.ridge_features(X, idx, off, np.arange(nt)), rtol=0, atol=2.5e-7)


# A float64 Gram matrix carries eps lambda_max, which a fit at penalty alpha feels as a few eps lambda_max /
# alpha of its norm: with at most 300 rows of 130 unit columns (lambda_max about 2,000 where half of them repeat) and
# alpha = 1e-3 some 1e-9 at worst.  The repository's bound for this search is 1e-8.
@pytest.mark.parametrize("noise", [1e-5, 1e-7, 1e-9, 0.0])
@pytest.mark.parametrize("nt,n", [(100, 100), (300, 130), (90, 130), (65, 64)])
def test_nearly_repeated_columns_at_a_small_penalty(gpu, noise, nt, n):
    """Columns that repeat others up to a little noise: singular values far below the largest, but above
    the rounding of X, count for the fit and its predictions; exactly repeated ones give no noise."""
    from hyperalignment_b200 import hyperalignment_c as H
    rng = np.random.default_rng(nt + n)
    ntot = nt + 40
    X = rng.standard_normal((ntot, n))
    X[:, n // 2:] = X[:, :n - n // 2] + noise * X[:, n // 2:]
    Y = X @ (0.1 * rng.standard_normal((n, n))) + rng.standard_normal((ntot, n))
    tr = [np.arange(nt, dtype=np.int32)]
    te = [np.arange(nt, ntot, dtype=np.int32)]
    sls = [np.arange(n, dtype=np.int32)]
    indptr, indices = H.sparse_pattern(sls, n)
    alphas, npcs = np.array([1e-3]), [n]
    data = np.zeros(indices.size)
    _, costs = H.searchlight_ridge_grid(X, Y, sls, indptr, indices, data, alphas, npcs, tr, te, return_costs=True)
    ref, _, rcosts = O.searchlight_ridge_grid_csc(X, Y, sls[0], np.array([0, n]), indptr, indices, np.zeros(indices.size),
                                                  alphas, npcs, tr, te, None)
    np.testing.assert_allclose(costs, rcosts, rtol=1e-8, atol=0)
    assert np.linalg.norm(data - ref) <= 1e-8 * np.linalg.norm(ref)


def test_grid_search_refuses_a_callers_stream_capture(gpu):
    """The search uploads lists from host memory that it frees: captured into a caller's graph, a replay would read
    freed memory.  The call fails instead (nothing is replayed here), and the plan works on afterwards."""
    import ctypes
    import torch
    rng = np.random.default_rng(3)
    n, nt = 20, 60
    X, Y = rng.standard_normal((nt, n)), rng.standard_normal((nt, n))
    plan = Plan(nt, n, np.arange(n), np.array([0, n]), weights=np.ones(n))
    dX, dY = upload(X), upload(Y)
    best = torch.zeros(1, dtype=torch.int32, device="cuda")
    vals = torch.zeros(plan.nnz, dtype=torch.float64, device="cuda")
    stream = torch.cuda.Stream()
    torch.cuda.synchronize()

    def run():
        plan.ridge_grid_device(dX.data_ptr(), dY.data_ptr(), vals.data_ptr(), best.data_ptr(), [1.0, 10.0], [5, n],
                               [np.arange(40)], [np.arange(40, nt)], stream=stream.cuda_stream)

    run()
    stream.synchronize()
    first = vals.cpu().numpy()
    rt = ctypes.CDLL("libcudart.so.12")
    rt.cudaStreamBeginCapture.argtypes = [ctypes.c_void_p, ctypes.c_int]
    rt.cudaStreamEndCapture.argtypes = [ctypes.c_void_p, ctypes.POINTER(ctypes.c_void_p)]
    graph = ctypes.c_void_p()
    assert rt.cudaStreamBeginCapture(stream.cuda_stream, 1) == 0  # thread-local mode
    try:
        with pytest.raises(RuntimeError):
            run()
    finally:
        rt.cudaStreamEndCapture(stream.cuda_stream, ctypes.byref(graph))
        rt.cudaGetLastError()
    vals.zero_()
    torch.cuda.synchronize()
    run()
    stream.synchronize()
    assert vals.cpu().numpy().tobytes() == first.tobytes()
    plan.close()
