"""Few block rows with many columns: the launch sequence, which splits the rows, or
the one launch.  The line is drawn by time; both sides give the solution, to
kappa(S) rtol of each other."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# 64 block rows of 17 blocks, 216 of 17, 512 of 17; columns on both sides of the line
@pytest.mark.parametrize("cells,b,one", [(2, 128, True), (2, 160, False), (2, 256, False), (3, 160, True), (3, 224, False),
                                         (4, 256, True)])
def test_line_between_the_stream_form_and_the_launch_sequence(cuda, cells, b, one):
    from kubomsd_b200 import lattices
    from tests.gpu_util import engine
    torch = cuda
    m = lattices.diamond_sp3(cells=cells, scale_hint=.24)
    S = m.S.tocsr()
    metric, _, _ = engine(m.H, S)
    cfg = metric._create[2]
    B = torch.randn((S.shape[0], b), dtype=torch.complex128, device="cuda")
    before = metric.lib.kmsd_kernel_launches()
    x, report = metric.solve(B, cfg)
    launches = metric.lib.kmsd_kernel_launches() - before
    assert report.converged.all() and (launches <= 3) == one
    narrow = torch.cat([metric.solve(B[:, j:j + 32].contiguous(), cfg)[0] for j in range(0, b, 32)], dim=1)
    lam = np.linalg.eigvalsh(S.toarray())
    bound = 1.01 * 2 * lam[-1] / lam[0] * 1e-10
    assert float(((x - narrow).norm(dim=0) / x.norm(dim=0)).max()) <= bound
