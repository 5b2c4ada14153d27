"""The metric solve as one launch (kmsd_pcg.cu) over its forms: one cluster, the
whole grid with the vectors in registers, and the whole grid with the vectors in
memory, at the edges of their column chunks and block-row shares.

A column that meets its threshold has |b - S x| <= rtol |b|, so its error is at
most kappa(S) rtol |x|; the solutions are held to that bound against a dense
solve, and the iteration counts to the oracle's within one (the rounding of the
recurrences differs)."""
import numpy as np
import pytest

from tests.test_gpu_segmented import atom_model

pytestmark = pytest.mark.gpu

RTOL = 1e-11


def _solve(S, blocks, B, policy="fixed", maxiter=1000, rtol=RTOL):
    from tests.gpu_util import engine
    metric, eng, _ = engine(S, S, blocks=blocks, rtol=rtol, policy=policy)
    cfg = metric._create[2]
    cfg.metric_maxiter = maxiter
    return metric, eng, cfg


# atoms, columns: 64 block rows is the smallest system of this path; 16 CTAs of
# 12 * 32 lanes hold 192 block rows of 32 columns, so 193 goes to the grid; more
# than 32 columns go in chunks and keep the vectors in memory
CASES = [(64, 1), (64, 4), (65, 5), (67, 8), (96, 9), (130, 16), (192, 32), (193, 32), (320, 17), (64, 33), (150, 64),
         (75, 100), (3000, 32)]


@pytest.mark.parametrize("na,b", CASES)
@pytest.mark.parametrize("cplx,pre,policy", [(False, "block", "fixed"), (True, "block", "fixed"),
                                             (False, "diagonal", "adaptive")])
def test_resident_solve(cuda, na, b, cplx, pre, policy):
    import scipy.sparse.linalg as sl
    from oracle import kpm_oracle as O
    H, S, blocks = atom_model(na, 7 * na + b, cplx=cplx)
    blocks = blocks if pre == "block" else []
    rng = np.random.default_rng(b)
    B = rng.standard_normal((S.shape[0], b)) + 1j * rng.standard_normal((S.shape[0], b))
    B *= np.logspace(-3, 3, b)
    if b > 3:
        B[:, 2] = 0.
    metric, eng, cfg = _solve(S, blocks, B, policy)
    x, report = metric.solve(B, cfg)
    want = sl.splu(S.tocsc()).solve(B)
    lam = sl.eigsh(S, k=1, which="LA", return_eigenvectors=False, tol=1e-6)[0], sl.eigsh(
        S, k=1, sigma=0., which="LM", return_eigenvectors=False, tol=1e-6)[0]
    bound = 1.01 * lam[0] / lam[1] * RTOL
    err, size = np.linalg.norm(x - want, axis=0), np.linalg.norm(want, axis=0)
    assert np.all(err <= bound * size), float(np.max(err / np.maximum(size, 1e-300)))
    assert report.converged.all()
    if na <= 320:
        ref = O.Metric(S, S.diagonal().real.copy(), blocks, policy).solve(B, RTOL, 0., 1000)[1]
        assert np.max(np.abs(report.iterations - np.asarray(ref["iterations"]))) <= 1
    # the engine's asynchronous solve is the same launch
    np.testing.assert_array_equal(eng.h_action(B), metric.solve(eng.H.matmul(B), cfg)[0])


def test_resident_solve_reports_failure(cuda):
    from kubomsd_b200.errors import NumericalError
    H, S, blocks = atom_model(80, 5)
    B = np.random.default_rng(0).standard_normal((S.shape[0], 6)) + 0j
    metric, eng, cfg = _solve(S, blocks, B, maxiter=2)
    with pytest.raises(NumericalError, match="true-residual acceptance") as info:
        metric.solve(B, cfg)
    assert info.value.diagnostics["iterations"] == [2] * 6
    assert not any(info.value.diagnostics["converged"])
    cfg.metric_maxiter = 1000
    x, report = metric.solve(B, cfg)  # the handle is usable after a failure
    assert report.converged.all()


def test_resident_solve_breakdown(cuda):
    import scipy.sparse as sp
    from kubomsd_b200.errors import NumericalError
    H, S, blocks = atom_model(80, 5)
    D = sp.diags(S.diagonal())
    B = np.random.default_rng(0).standard_normal((S.shape[0], 6)) + 0j
    metric, eng, cfg = _solve((D + 60. * (S - D)).tocsr(), [], B)  # indefinite, positive diagonal
    with pytest.raises(NumericalError, match="curvature breakdown"):
        metric.solve(B, cfg)


@pytest.mark.parametrize("b", [8, 32])
def test_first_solves_of_replicas_behind_large_copies(cuda, b):
    """Block patterns and counters that a replica's first solve uploads are on
    the device before its kernel runs, also while other streams keep the copy
    engine busy; the solves are deterministic, so all agree bit for bit."""
    import threading
    import torch
    from tests.gpu_util import engine
    H, S, blocks = atom_model(400, 5)
    metric, eng, _ = engine(H, S, blocks=blocks, rtol=RTOL)
    rng = np.random.default_rng(b)
    B = torch.from_numpy(rng.standard_normal((S.shape[0], b)) + 0j).cuda()
    want = eng.h_action(B).cpu()
    replicas = [eng.replica() for _ in range(4)]
    host = torch.empty(1 << 28, dtype=torch.uint8).pin_memory()
    dev = torch.empty(1 << 28, dtype=torch.uint8, device="cuda")
    copies = torch.cuda.Stream()
    torch.cuda.synchronize()
    got = [None] * len(replicas)

    def first(i):
        with torch.cuda.stream(torch.cuda.Stream()):
            got[i] = replicas[i].h_action(B).cpu()

    with torch.cuda.stream(copies):
        for _ in range(8):
            dev.copy_(host, non_blocking=True)
    threads = [threading.Thread(target=first, args=(i,)) for i in range(len(replicas))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    for x in got:
        assert torch.equal(x, want)
