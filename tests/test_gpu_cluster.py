"""Moments of small operators in one launch (kmsd_cluster.cu) against the oracle,
at the edges of its row shares, row widths, column groups and sum histories.

Tolerances are the path's own: 1e-10 of the largest moment in FP64, 5e-5 in the
mixed form (complex64 vectors)."""
import numpy as np
import pytest
import scipy.sparse as sp

from tests.helpers import assert_rel

pytestmark = pytest.mark.gpu


def ring(n, reach, seed):
    """A Hermitian real operator with up to 2 reach + 1 entries per row: rows are
    short at random, so that padding is used."""
    rng = np.random.default_rng(seed)
    A = sp.diags([rng.uniform(-.5, .5, n)], [0]).tolil() if n < 40 else sp.diags([rng.uniform(-.5, .5, n)], [0])
    A = A.tocsr()
    for d in range(1, reach + 1):
        i = np.arange(n)
        j = (i + d * d * 7) % n
        keep = (rng.random(n) < .9) & (i != j)
        B = sp.coo_matrix((np.full(keep.sum(), -1. / d), (i[keep], j[keep])), shape=(n, n)).tocsr()
        A = A + B + B.T
    A = A.tocsr()
    A.sum_duplicates()
    return A


# rows, reach (width 3, 5, 7), columns, moments
CASES = [(1, 1, 1, 3), (5, 1, 2, 2), (33, 1, 3, 64), (480, 2, 1, 65), (481, 2, 4, 66), (1000, 3, 5, 129), (4096, 2, 8, 130),
         (9729, 1, 6, 33), (15361, 3, 2, 20), (15360, 3, 33, 9), (20011, 2, 9, 12), (30720, 2, 3, 9), (38912, 1, 2, 9)]


@pytest.mark.parametrize("n,reach,b,M", CASES)
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("doubling", [False, True])
def test_cluster_moments(cuda, n, reach, b, M, precision, doubling):
    from oracle import kpm_oracle as O
    from tests.gpu_util import engine
    H = ring(n, reach, n + b)
    S = sp.identity(n, format="csr")
    _, eng, _ = engine(H, S, precision=precision)
    half = 1.05 * float(abs(H).sum(axis=1).max()) + .1
    B = np.exp(2j * np.pi * np.random.default_rng(b).random((n, b)))
    lib = eng.lib
    before = lib.kmsd_kernel_launches()
    got = eng.moments(B, M, .05, half, doubling=doubling)
    launches = lib.kmsd_kernel_launches() - before
    limit = 16 * (480 if precision == "fp64" else 608) * (4 if H.indptr.size and np.diff(H.indptr).max() < 6 else 2)
    if n <= limit:
        assert launches == 2  # the finiteness check of B and the moments
    want = O.engine_from_model(H, S).moments(B, M, .05, half)
    assert_rel(got, want, 1e-10 if precision == "fp64" else 5e-5, f"{n} {b} {M}")
    np.testing.assert_array_equal(got, eng.moments(B, M, .05, half, doubling=doubling))
    assert eng.core.h_calls == 2 * ((M + 1) // 2 if doubling else M - 1)


def test_complex_and_wide_rows_keep_the_launch_per_step(cuda):
    from oracle import kpm_oracle as O
    from tests.gpu_util import engine
    n = 500
    S = sp.identity(n, format="csr")
    B = np.exp(2j * np.pi * np.random.default_rng(1).random((n, 3)))
    H = ring(n, 2, 1).astype(complex)
    H = H + 1j * (sp.triu(ring(n, 1, 2), 1) - sp.tril(ring(n, 1, 2), -1))
    for A in (H.tocsr(), ring(n, 6, 3)):
        _, eng, _ = engine(A, S)
        half = 1.05 * float(abs(A).sum(axis=1).max())
        want = O.engine_from_model(A, S).moments(B, 40, 0., half)
        assert_rel(eng.moments(B, 40, 0., half), want, 1e-10)


@pytest.mark.parametrize("precision,doubling", [("fp64", False), ("fp64", True), ("mixed", False), ("mixed", True)])
@pytest.mark.parametrize("sizes,b,M", [((1, 40, 700, 33), 5, 70), ((600, 5000, 20011, 64, 97), 9, 12), ((300,) * 20, 2, 66)])
def test_cluster_batch(cuda, sizes, b, M, precision, doubling):
    # every instance with its own window, all in one launch, against separate calls
    from kubomsd_b200.batch import B200Batch
    from tests.gpu_util import engine
    Hs = [ring(n, 2, 50 + i) for i, n in enumerate(sizes)]
    halves = [1.05 * float(abs(H).sum(axis=1).max()) + .1 for H in Hs]
    centers = [.01 * i for i in range(len(sizes))]
    rng = np.random.default_rng(b)
    Bs = [np.exp(2j * np.pi * rng.random((n, b))) for n in sizes]
    bt = B200Batch(Hs, precision=precision)
    before = bt.lib.kmsd_kernel_launches()
    got = bt.moments(Bs, M, centers, halves, doubling=doubling).cpu().numpy()
    assert bt.lib.kmsd_kernel_launches() - before == 1
    for i, H in enumerate(Hs):
        _, eng, _ = engine(H, sp.identity(sizes[i], format="csr"), precision=precision)
        want = eng.moments(Bs[i], M, centers[i], halves[i], doubling=doubling)
        # the same elements, the FP64 sums in another order
        assert_rel(got[i], want, 1e-13, f"instance {i}")


def velocity_of(H, seed, drop=0.):
    """A purely imaginary Hermitian velocity on (part of) H's off-diagonal pattern."""
    U = sp.triu(H, 1).tocoo()
    rng = np.random.default_rng(seed)
    w = rng.uniform(.2, 1., U.nnz) * (rng.random(U.nnz) >= drop)
    A = sp.coo_matrix((1j * U.data * w, (U.row, U.col)), shape=H.shape).tocsr()
    A.eliminate_zeros()
    return (A + A.conj().T).tocsr()


# rows, reach, psi columns, directions: shares of 480 / 608 rows and their doubles,
# no phi block, one and two directions, one with a velocity outside one axis
@pytest.mark.parametrize("n,reach,nb,dirs", [(7, 1, 2, [[1., 0., 0.]]), (480, 2, 4, [[1., 0., 0.]]), (4096, 2, 8, []),
                                             (1000, 3, 6, [[1., 0., 0.], [0., -1., 0.]]), (9729, 2, 2, [[0., 2., 0.]]),
                                             (15360, 2, 34, [[1., 0., 0.]]), (4096, 1, 2, [[.6, .8, 0.]])])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_cluster_series(cuda, n, reach, nb, dirs, precision):
    from oracle import kpm_oracle as O
    from tests.gpu_util import engine
    H = ring(n, reach, n + nb)
    V = {"x": velocity_of(H, 1), "y": velocity_of(H, 2, .5)}
    S = sp.identity(n, format="csr")
    half = 1.05 * float(abs(H).sum(axis=1).max()) + .1
    rng = np.random.default_rng(n)
    b = nb * (1 + len(dirs))
    B = rng.standard_normal((n, b)) + 1j * rng.standard_normal((n, b))
    _, eng, _ = engine(H, S, velocity=V, precision=precision)
    ref = O.engine_from_model(H, S, velocity=V)
    for terms in (2, 3, 40):
        coeff = (rng.standard_normal(terms) + 1j * rng.standard_normal(terms)) * .8 ** np.arange(terms)
        before = eng.lib.kmsd_kernel_launches()
        got = eng.series(B, coeff, .03, half, dirs)
        launches = eng.lib.kmsd_kernel_launches() - before
        if all(np.count_nonzero(d) == 1 and V["xy"[np.argmax(np.abs(d))]].nnz for d in dirs):
            assert launches == 1 + max(1, len(dirs))  # the finiteness check of B, then one per direction
        assert_rel(got, ref.series(B, coeff, .03, half, dirs), 1e-10 if precision == "fp64" else 5e-5, f"{terms}")
    assert eng.core.h_calls == 1 + 2 + 39 and eng.core.v_calls == 42 * len(dirs)


def test_cluster_series_reports_nonfinite(cuda):
    from kubomsd_b200.errors import NumericalError
    from tests.gpu_util import engine
    H = ring(300, 2, 9)
    _, eng, _ = engine(H, sp.identity(300, format="csr"))
    B = np.ones((300, 2), complex)
    with pytest.raises(NumericalError, match="nonfinite Chebyshev propagation"):
        eng.series(B, np.ones(150), 0., 1e-3)  # far outside the window: T_k overflows


@pytest.mark.parametrize("n,reach,b,length", [(7, 1, 2, 2), (480, 2, 4, 33), (3000, 3, 6, 5), (15361, 1, 2, 4), (1000, 2, 34, 3)])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_cluster_chain(cuda, n, reach, b, length, precision):
    from oracle import kpm_oracle as O
    from tests.gpu_util import engine
    H = ring(n, reach, n + b)
    S = sp.identity(n, format="csr")
    half = 1.05 * float(abs(H).sum(axis=1).max()) + .1
    rng = np.random.default_rng(n)
    B = rng.standard_normal((n, b)) + 1j * rng.standard_normal((n, b))
    _, eng, _ = engine(H, S, precision=precision)
    got = eng.chain(B, length, .03, half)
    assert_rel(got, O.engine_from_model(H, S).chain(B, length, .03, half), 1e-10 if precision == "fp64" else 5e-5)
    assert eng.core.h_calls == length - 1
    # the same chain through the ring of the correlation tables, against cov = B
    cov = np.ascontiguousarray(np.broadcast_to(B[:, None, :], (n, 1, b)))
    tables = eng.chain_correlate(B, cov, length, .03, half).cpu().numpy()[:, :, 0]
    want = np.einsum("jnb,nb->bj", got.conj(), B)
    assert np.all(abs(tables - want) <= 1e-12 * np.einsum("jnb,nb->bj", abs(got), abs(B)))
