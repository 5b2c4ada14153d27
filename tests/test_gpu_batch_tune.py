"""The batch tuner sweeps tile sizes where there are tiles, and only there."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tiles", [False, True])
def test_tuner_sweeps_only_where_there_are_tiles(cuda, tiles):
    import numpy as np
    from kubomsd_b200 import kpm, lattices
    from kubomsd_b200.batch import B200Batch
    # 180 x 180 sites do not fit a cluster
    ms = [lattices.square_lattice(s, seed=s) for s in ((24, 180) if tiles else (24, 40))]
    B = cuda.from_numpy(np.concatenate([kpm.random_phases(m.n, 3, range(4)) for m in ms])).cuda()
    bt = B200Batch([m.H for m in ms], precision="fp64", tile_rows=700)
    want = bt.moments(B, 12, 0., 12., doubling=False).clone()
    before = bt.lib.kmsd_kernel_launches()
    rows = bt._tune_rows(B, 12, [0., 0.], [12., 12.], False)
    launches = bt.lib.kmsd_kernel_launches() - before
    if tiles:
        assert rows in (512, 1024, 2048, 4096, 8192) and launches == 10 * 22  # a step and a reduction each
    else:
        assert rows == 700 and launches == 1
    # sums of other tiles round differently
    assert float((bt.moments(B, 12, 0., 12., doubling=False) - want).abs().max()) <= 1e-12 * float(want.abs().max())
