"""Stored chains on both sides of the line between one launch of clusters and a
launch per step: the same chain as the oracle's."""
import numpy as np
import pytest
import scipy.sparse as sp

from tests.helpers import assert_rel
from tests.test_gpu_cluster import ring

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision,reach,b,one", [("fp64", 2, 206, True), ("fp64", 2, 208, False), ("fp64", 3, 122, True),
                                                   ("fp64", 3, 123, False), ("mixed", 3, 206, True), ("mixed", 3, 208, False)])
def test_chain_on_both_sides_of_the_line(cuda, precision, reach, b, one):
    from oracle import kpm_oracle as O
    from tests.gpu_util import engine
    n, length = 4096, 5
    H, S = ring(n, reach, 3), sp.identity(4096, format="csr")
    _, eng, _ = engine(H, S, precision=precision)
    half = 1.1 * float(abs(H).sum(axis=1).max())
    B = np.exp(2j * np.pi * np.random.default_rng(b).random((n, b)))
    before = eng.lib.kmsd_kernel_launches()
    got = eng.chain(B, length, .05, half)
    assert (eng.lib.kmsd_kernel_launches() - before <= 2) == one
    want = O.engine_from_model(H, S).chain(B, length, .05, half)
    assert_rel(got, want, 1e-10 if precision == "fp64" else 5e-5, f"{b}")
