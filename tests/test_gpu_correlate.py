"""The correlation tables (kmsd_engine_chain_correlate) against the contraction of
the engine's own stored chain, at the edges of the ring (32 vectors), the thread
tiles (8 vectors x 4 terms), the k tiles and the row chunks and stages.

Both are FP64 sums of n products in different orders: they differ by at most
2 n eps times the sum of the moduli, far below 1e-12 of it for these n."""
import numpy as np
import pytest
import scipy.sparse as sp

from tests.test_gpu_cluster import ring

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,b,length,kcols", [(1, 1, 1, 1), (7, 3, 33, 5), (149, 8, 32, 41), (300, 5, 40, 44),
                                              (1000, 8, 71, 45), (2500, 4, 64, 97), (513, 1, 10, 353), (400, 2, 31, 4),
                                              (5000, 7, 9, 128), (50, 8, 35, 128)])
def test_tables_equal_the_contracted_chain(cuda, n, b, length, kcols):
    from tests.gpu_util import engine
    H = ring(n, 2, n)
    _, eng, _ = engine(H, sp.identity(n, format="csr"))
    half = 1.05 * float(abs(H).sum(axis=1).max()) + .1
    rng = np.random.default_rng(n + b)
    B = rng.standard_normal((n, b)) + 1j * rng.standard_normal((n, b))
    cov = rng.standard_normal((n, kcols, b)) + 1j * rng.standard_normal((n, kcols, b))
    tables = eng.chain_correlate(B, cov, length, 0., half).cpu().numpy()
    chain = eng.chain(B, length, 0., half)
    want = np.einsum("jnb,nkb->bjk", chain.conj(), cov)
    scale = np.einsum("jnb,nkb->bjk", abs(chain), abs(cov))
    assert np.all(abs(tables - want) <= 1e-12 * scale + 1e-300)
    np.testing.assert_array_equal(tables, eng.chain_correlate(B, cov, length, 0., half).cpu().numpy())
