"""A handle is valid on any stream once its constructor has returned: uploads and
clears that went through the legacy stream are on the device by then, also while
other streams keep the copy engines busy.  Every object here is made and first used
inside a non-blocking stream behind large copies."""
from contextlib import contextmanager

import numpy as np
import pytest

from tests.test_gpu_segmented import atom_model

pytestmark = pytest.mark.gpu


@contextmanager
def _busy(torch):
    host = torch.empty(1 << 27, dtype=torch.uint8).pin_memory()
    dev = torch.empty(1 << 27, dtype=torch.uint8, device="cuda")
    copies, work = torch.cuda.Stream(), torch.cuda.Stream()
    torch.cuda.synchronize()
    with torch.cuda.stream(copies):
        for _ in range(8):
            dev.copy_(host, non_blocking=True)
    with torch.cuda.stream(work):
        yield
    torch.cuda.synchronize()


@pytest.mark.parametrize("side", [30, 150])
def test_first_moments_of_a_lattice(cuda, side):
    from kubomsd_b200 import kpm, lattices
    from tests.gpu_util import engine
    m = lattices.square_lattice(side, seed=side)
    B = cuda.from_numpy(kpm.random_phases(m.n, 1, range(4))).cuda()
    with _busy(cuda):
        _, eng, _ = engine(m.H, m.S)
        first = eng.moments(B, 16, 0., 12.).cpu()
    assert cuda.equal(first, eng.moments(B, 16, 0., 12.).cpu())


@pytest.mark.parametrize("nb", [4, 3])  # one launch; the launch sequence
def test_first_solve_of_a_metric(cuda, nb):
    from tests.gpu_util import engine
    H, S, blocks = atom_model(200, 3, nb=nb)
    B = cuda.from_numpy(np.random.default_rng(0).standard_normal((S.shape[0], 6)) + 0j).cuda()
    with _busy(cuda):
        metric, eng, _ = engine(H, S, blocks=blocks)
        first = metric.solve(B, metric._create[2])[0].cpu()
    assert cuda.equal(first, metric.solve(B, metric._create[2])[0].cpu())


def test_first_call_of_a_segmented_batch(cuda):
    from kubomsd_b200.batch import B200Batch
    models = [atom_model(na, na) for na in (20, 33, 70)]
    n = sum(H.shape[0] for H, _, _ in models)
    B = cuda.from_numpy(np.random.default_rng(0).standard_normal((n, 4)) + 0j).cuda()
    with _busy(cuda):
        bt = B200Batch([H for H, _, _ in models], precision="fp64", overlaps=[S for _, S, _ in models],
                       blocks=[b for _, _, b in models])
        first = bt.moments(B, 6, 0., 60.).cpu()
    assert cuda.equal(first, bt.moments(B, 6, 0., 60.).cpu())
    bt2 = B200Batch([H for H, _, _ in models], precision="mixed")
    with _busy(cuda):
        assert bt2.lib.kmsd_batch_set_tile_rows(bt2.handle, 64) == 0
        first = bt2.moments(B, 1, 0., 60.).cpu()  # one moment: the tile kernels
    assert cuda.equal(first, bt2.moments(B, 1, 0., 60.).cpu())
