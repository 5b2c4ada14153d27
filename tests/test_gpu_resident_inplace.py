"""kmsd_metric_solve with the solution written over its right-hand side.

The one-launch solve reads the right-hand side again wherever it forms a true
residual.  Near the attainable accuracy a few columns of a thousand leave by the
recurrence's residual with a true residual just above the threshold and go on, so
these solves read it after an acceptance too; over 8,000 columns some do in every
form."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _diamond():
    from kubomsd_b200 import lattices
    from tests.gpu_util import engine
    m = lattices.diamond_sp3(cells=4, scale_hint=.24)
    S = m.S.tocsr()
    blocks = [(i, j, np.linalg.cholesky(S[i:j, i:j].toarray())) for i, j in m.atom_slices]
    metric, _, _ = engine(m.H, S, blocks=blocks)
    return metric, S


def _solve(torch, metric, x, y, rtol):
    return metric.lib.kmsd_metric_solve(metric.handle, C.c_void_p(x.data_ptr()), C.c_void_p(y.data_ptr()), x.shape[1],
                                        rtol, 0., 1000, None, C.c_void_p(torch.cuda.current_stream().cuda_stream))


# one cluster; the grid with the vectors in registers; the grid with the vectors in memory
@pytest.mark.parametrize("b", [8, 32, 64])
def test_solution_over_its_right_hand_side(cuda, b):
    torch = cuda
    metric, S = _diamond()
    g = torch.Generator(device="cuda").manual_seed(b)
    for _ in range(8000 // b):
        B = torch.randn((S.shape[0], b), dtype=torch.complex128, device="cuda", generator=g)
        apart, over = torch.empty_like(B), B.clone()
        rc = _solve(torch, metric, B, apart, 1e-14)
        assert _solve(torch, metric, over, over, 1e-14) == rc  # (a column may miss for good, then in both)
        if rc == 0:
            assert torch.equal(over, apart)


@pytest.mark.parametrize("b", [8, 32, 64])
def test_columns_that_just_miss_go_on(cuda, b):
    """A column above its threshold by less than the threshold itself goes on and
    converges, and the solve is counted (kmsd_metric_stats.refinement_steps); one that
    is further off fails the solve with its residual."""
    from kubomsd_b200.errors import NumericalError
    torch = cuda
    rtol = 1e-14
    metric, S = _diamond()
    cfg = metric._create[2]
    cfg.metric_rtol = rtol
    A = torch.sparse_csr_tensor(torch.from_numpy(S.indptr.astype(np.int64)), torch.from_numpy(S.indices.astype(np.int64)),
                                torch.from_numpy(S.data.astype(complex)), size=S.shape).cuda()
    g = torch.Generator(device="cuda").manual_seed(b)
    for _ in range(8000 // b):
        B = torch.randn((S.shape[0], b), dtype=torch.complex128, device="cuda", generator=g)
        try:
            x, report = metric.solve(B, cfg)
        except NumericalError as exc:
            rel = np.array(exc.diagnostics["relative_residual"])
            assert rel[~np.array(exc.diagnostics["converged"])].min() > 2 * rtol * (1 - 1e-9)
            continue
        assert report.converged.all() and report.relative_residual.max() <= rtol * (1 + 1e-9)
        # formed once more, with roundings of about a hundredth of the threshold at most
        assert float(((B - A @ x).norm(dim=0) / B.norm(dim=0)).max()) <= 1.1 * rtol
    assert metric.stats().refinement_steps > 0
