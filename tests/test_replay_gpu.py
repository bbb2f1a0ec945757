"""Captured graphs against direct launches, and the per-phase tensor-core iteration with its own switches
(HA_B200_TC_RESIDENT=0: by default the resident and the wide kernels take every searchlight)."""

import os
import subprocess
import sys

import numpy as np
import pytest

from hyperalignment_b200 import _lib as L
from hyperalignment_b200 import workloads as W
from hyperalignment_b200.plan import Plan

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def upload(X):
    import torch
    return torch.from_numpy(np.asfortranarray(X).ravel(order="F")).cuda()


def test_wide_iteration_graph_matches_direct_launches(gpu, hlib):
    """Searchlights of more than 256 vertices run in the captured loop, the others beside it on the side streams:
    the capturing call, replays, a new output order (captured again) and new data in the same buffers give the
    bits of direct launches."""
    import torch
    rng = np.random.default_rng(4)
    nt, nv = 500, 420
    sizes = [200, 257, 300, 128, 400, 40, 256, 272]
    idx = np.concatenate([np.sort(rng.choice(nv, n, replace=False)) for n in sizes]).astype(np.int32)
    off = np.concatenate([[0], np.cumsum(sizes)]).astype(np.int32)
    data = []
    for _ in range(2):
        X = rng.standard_normal((nt, nv))
        data.append((upload(X), upload(X @ np.linalg.qr(rng.standard_normal((nv, nv)))[0] + 0.1 * rng.standard_normal((nt, nv)))))
    plan = Plan(nt, nv, idx, off, weights=np.ones(idx.size))
    dX, dY = torch.empty_like(data[0][0]), torch.empty_like(data[0][1])
    vals = torch.zeros(plan.nnz, dtype=torch.float64, device="cuda")

    def run(which, kind):
        dX.copy_(data[which][0])
        dY.copy_(data[which][1])
        vals.zero_()
        plan.procrustes_device(dX.data_ptr(), dY.data_ptr(), vals.data_ptr(), True, True, L.SOLVER_TC, kind)
        torch.cuda.synchronize()
        return vals.cpu().numpy().tobytes()

    calls = [(0, L.OUT_CSC), (0, L.OUT_CSC), (1, L.OUT_CSC), (1, L.OUT_CSR), (0, L.OUT_CSR), (0, L.OUT_CSC)]
    try:
        hlib.ha_b200_set_graphs(False)
        direct = [run(*c) for c in calls]
        hlib.ha_b200_set_graphs(True)
        graph = [run(*c) for c in calls]
    finally:
        hlib.ha_b200_set_graphs(True)
        plan.close()
    assert graph == direct
    assert len(set(direct)) == 4  # two data sets, two orders


def test_fp32_grid_graph_matches_direct_launches(gpu, hlib):
    """The plain FP32 grid search (the form that is captured) over changing penalties, PC counts and folds, and with
    new data in the same buffers: replays and new captures give the bits of direct launches."""
    import torch
    from hyperalignment_b200 import hyperalignment_c as H
    w = W.small_case(seed=8, nv=642, nt=120, lo=10, hi=60)
    rng = np.random.default_rng(1)
    plan = Plan(w.nt, w.nv, w.sls.indices, w.sls.offsets, w.sls.dists, w.sls.radius)
    plan.set_grid_precision(32)
    Ys = [upload(0.5 * w.Y + rng.standard_normal(w.Y.shape)) for _ in range(2)]
    dX, dY = upload(w.X), torch.empty_like(Ys[0])
    folds = [H.ensemble_indices(120, 1, f, 6, 3, 4) for f in (5, 4)]
    vals = torch.zeros(plan.nnz, dtype=torch.float64, device="cuda")
    best = torch.zeros(w.sls.count, dtype=torch.int32, device="cuda")
    cost = torch.zeros(w.sls.count * 12, dtype=torch.float64, device="cuda")

    def run(y, fold, alphas, npcs):
        dY.copy_(Ys[y])
        vals.zero_()
        best.fill_(-1)
        cost.zero_()
        plan.ridge_grid_device(dX.data_ptr(), dY.data_ptr(), vals.data_ptr(), best.data_ptr(), alphas, npcs, *folds[fold],
                               d_cost=cost.data_ptr())
        torch.cuda.synchronize()
        return vals.cpu().numpy().tobytes(), best.cpu().numpy().tobytes(), cost.cpu().numpy().tobytes()

    a = (np.logspace(-3, 3, 4), [5, 10, 40])
    b = (np.logspace(-2, 2, 4), [5, 10, 40])  # same shape, other penalties
    c = (np.logspace(-2, 2, 3), [5, 10, 40, 1 << 30])
    calls = [(0, 0, *a), (0, 0, *a), (1, 0, *a), (0, 0, *b), (0, 0, *c), (0, 1, *c), (0, 0, *a)]
    try:
        hlib.ha_b200_set_graphs(False)
        direct = [run(*x) for x in calls]
        hlib.ha_b200_set_graphs(True)
        graph = [run(*x) for x in calls]
    finally:
        hlib.ha_b200_set_graphs(True)
        plan.close()
    assert graph == direct
    assert len(set(direct)) == 5


_PHASE_SCRIPT = r"""
import sys
import numpy as np
import torch
sys.path.insert(0, sys.argv[1])
from hyperalignment_b200 import _lib as L
from hyperalignment_b200.plan import Plan
rng = np.random.default_rng(6)
sizes = [40, 64, 100, 128, 129, 200, 256, 257, 300]
nv, nt = 300, 400
X = rng.standard_normal((nt, nv))
Y = X @ np.linalg.qr(rng.standard_normal((nv, nv)))[0] + 0.1 * rng.standard_normal((nt, nv))
X[:, 7] = X[:, 3]
idx = np.concatenate([np.arange(n) for n in sizes]).astype(np.int32)
off = np.concatenate([[0], np.cumsum(sizes)]).astype(np.int32)
plan = Plan(nt, nv, idx, off, weights=np.ones(idx.size))
dX = torch.from_numpy(np.asfortranarray(X).ravel(order="F")).cuda()
dY = torch.from_numpy(np.asfortranarray(Y).ravel(order="F")).cuda()
v = torch.zeros(plan.nnz, dtype=torch.float64, device="cuda")
out = []
for layout in eval(sys.argv[3]):
    if layout is not None:
        plan.set_tc_layout(layout)
    v.zero_()
    plan.procrustes_device(dX.data_ptr(), dY.data_ptr(), v.data_ptr(), True, True, L.SOLVER_TC, L.OUT_CSR)
    out.append(v.cpu().numpy())
np.save(sys.argv[2], np.stack(out))
"""


def _phase_run(path, layouts="[None]", **env):
    subprocess.run([sys.executable, "-c", _PHASE_SCRIPT, ROOT, str(path), layouts], env=dict(os.environ, **env), check=True,
                   timeout=300)
    return [a.tobytes() for a in np.load(path)]


def test_per_phase_layouts_bitwise_equal(gpu, tmp_path):
    """The per-phase launches under the tuned and every kind of pinned layout: the bits of the default kernels."""
    default = _phase_run(tmp_path / "d.npy")[0]
    outs = _phase_run(tmp_path / "l.npy", "[None, (110, 110), (53, 200), (72, 110)]", HA_B200_TC_RESIDENT="0")
    assert all(o == default for o in outs)


def test_per_phase_switch_point_bitwise_equal(gpu, tmp_path):
    """The per-phase launches, the persistent kernel taking over always, from iteration 5 or never, captured or
    launched one by one: the bits of the default kernels."""
    default = _phase_run(tmp_path / "d.npy")[0]
    for first, graphs in (("0", "1"), ("5", "0"), ("1000", "1")):
        out = _phase_run(tmp_path / f"f{first}.npy", "[None, None]", HA_B200_TC_RESIDENT="0", HA_B200_TC_ITER_FROM=first,
                         HA_B200_GRAPHS=graphs)
        assert all(o == default for o in out), (first, graphs)
