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
