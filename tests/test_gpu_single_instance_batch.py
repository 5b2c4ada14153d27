"""A nonorthogonal batch of one instance: its solves are one launch each, recorded in
the batch's graph; other column counts grow the buffers and are recorded anew."""
import numpy as np
import pytest

from tests.helpers import assert_rel
from tests.test_gpu_segmented import atom_model

pytestmark = pytest.mark.gpu


# one cluster; the grid; the grid with the vectors in memory
@pytest.mark.parametrize("na", [70, 400])
@pytest.mark.parametrize("storage", ["fp64", "mixed"])
def test_batch_of_one_nonorthogonal_instance(cuda, na, storage):
    from kubomsd_b200.batch import B200Batch
    from tests.gpu_util import engine
    H, S, blocks = atom_model(na, 2)
    half = 1.1 * float(abs(H).sum(axis=1).max())
    _, eng, _ = engine(H, S, blocks=blocks)
    bt = B200Batch([H], precision=storage, overlaps=[S], blocks=[blocks])
    rng = np.random.default_rng(na)
    for b in (5, 40, 5, 20):
        x = rng.standard_normal((H.shape[0], b)) + 1j * rng.standard_normal((H.shape[0], b))
        B = cuda.from_numpy(x).cuda()
        calls = [bt.moments(B, 7, 0., half, use_graph=g).cpu().numpy() for g in (True, True, False)]
        for got in calls[1:]:
            np.testing.assert_array_equal(got, calls[0])
        # both solve to 1e-10 with kappa(S) below 10, eight times in a row
        assert_rel(calls[0][0], eng.moments(x, 7, 0., half), 1e-8, f"{na} {b}")
