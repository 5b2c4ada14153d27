"""The paths that serve what the one-launch cluster kernels decline: larger lattices,
rows of more than eight entries, complex Hamiltonians, velocities with a real part.
Small systems reach those kernels only through the last three."""
import numpy as np
import pytest
import scipy.sparse as sp

from tests.helpers import assert_rel
from tests.test_gpu_cluster import ring

pytestmark = pytest.mark.gpu

TOL = {"fp64": 1e-10, "mixed": 5e-5}


def _twisted(H, seed):
    """H with phases on its bonds: complex, Hermitian, the same pattern."""
    U = sp.triu(sp.csr_matrix(H), 1).tocoo()
    w = U.data * np.exp(1j * np.random.default_rng(seed).uniform(-1, 1, U.nnz))
    T = sp.coo_matrix((w, (U.row, U.col)), shape=H.shape).tocsr()
    return (T + T.conj().T + sp.diags(H.diagonal())).tocsr()


def _instances(kind):
    from kubomsd_b200 import lattices
    small = [lattices.honeycomb(9, 7, seed=1, with_velocity=False).H, lattices.honeycomb(31, 20, seed=2, with_velocity=False).H]
    if kind == "rows":  # 41,402 rows of four entries: an ELL form for the whole batch
        return small + [lattices.honeycomb(163, 127, seed=3, with_velocity=False).H]
    if kind == "wide":
        return small + [ring(517, 6, 4)]
    return small + [_twisted(small[1], 5)]


@pytest.mark.parametrize("kind", ["rows", "wide", "complex"])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("doubling", [False, True])
def test_batch_of_instances_beyond_a_cluster(cuda, kind, precision, doubling):
    from kubomsd_b200.batch import B200Batch
    from tests.gpu_util import engine
    Hs = _instances(kind)
    n, M = sum(H.shape[0] for H in Hs), 21
    half = [1.1 * float(abs(H).sum(axis=1).max()) for H in Hs]
    center = [.1 * i for i in range(len(Hs))]
    bt = B200Batch(Hs, precision=precision, tile_rows=700)
    steps = (M + 1) // 2 if doubling else M - 1
    rng = np.random.default_rng(n)
    kept = {}
    for b in (3, 8, 3):  # the second grows the buffers: the first graph is recorded anew
        if b not in kept:
            x = np.exp(2j * np.pi * rng.random((n, b)))
            kept[b] = x, cuda.from_numpy(x).cuda(), None
        x, B, first = kept[b]
        calls = []
        for _ in range(3):  # recorded, replayed, replayed
            before = bt.lib.kmsd_kernel_launches()
            calls.append(bt.moments(B, M, center, half, doubling=doubling).cpu().numpy())
            assert bt.lib.kmsd_kernel_launches() - before >= 2 * steps
        direct = bt.moments(B, M, center, half, doubling=doubling, use_graph=False).cpu().numpy()
        for got in calls[1:] + [direct] + ([first] if first is not None else []):
            np.testing.assert_array_equal(got, calls[0])
        kept[b] = x, B, calls[0]
        for i, H in enumerate(Hs):
            _, eng, _ = engine(H, sp.identity(H.shape[0], format="csr"), precision=precision)
            part = x[bt.offsets[i]:bt.offsets[i + 1]]
            assert_rel(calls[0][i], eng.moments(part, M, center[i], half[i], doubling=doubling), 1e-10, f"{kind} {i} {b}")


@pytest.mark.parametrize("case", ["honeycomb", "square", "width 12", "width 13", "complex"])
@pytest.mark.parametrize("b", [1, 3, 17])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("doubling", [False, True])
def test_moments_beyond_a_cluster(cuda, case, b, precision, doubling):
    from kubomsd_b200 import lattices
    from oracle import kpm_oracle as O
    from tests.gpu_util import engine
    H = {"honeycomb": lambda: lattices.honeycomb(163, 127, seed=3, with_velocity=False).H,  # odd sides, ELL of width 4
         "square": lambda: lattices.square_lattice(201, seed=4).H,  # rows of five: CSR
         "width 12": lambda: ring(263, 5, 6), "width 13": lambda: ring(97, 6, 7),
         "complex": lambda: _twisted(ring(130, 1, 8), 9)}[case]()
    n, M = H.shape[0], 10
    S = sp.identity(n, format="csr")
    half = 1.1 * float(abs(H).sum(axis=1).max())
    _, eng, _ = engine(H, S, precision=precision)
    B = np.exp(2j * np.pi * np.random.default_rng(b).random((n, b)))
    before = eng.lib.kmsd_kernel_launches()
    got = eng.moments(B, M, .05, half, doubling=doubling)
    assert eng.lib.kmsd_kernel_launches() - before >= ((M + 1) // 2 if doubling else M - 1)
    assert_rel(got, O.engine_from_model(H, S).moments(B, M, .05, half), TOL[precision], f"{case} {b}")


@pytest.mark.parametrize("velocity,R", [("complex", 2), ("complex", 16), ("complex", 32), ("complex", 64), ("imaginary", 2),
                                        ("imaginary", 18)])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_series_beyond_a_cluster(cuda, velocity, R, precision):
    """[psi | phi] with V on H's pattern, in row groups of 4 to 128 lanes: V with real
    and imaginary parts on a small lattice, and purely imaginary, whose real plane is
    not read, on one of 41,402 sites."""
    from kubomsd_b200 import kpm, lattices
    from kubomsd_b200.config import RunConfig
    from oracle import kpm_oracle as O
    from tests.gpu_util import engine
    m = lattices.honeycomb(13, 11, seed=8) if velocity == "complex" else lattices.honeycomb(163, 127, seed=8)
    V = m.velocity["x"] if velocity == "imaginary" else _twisted(m.H, 3)
    B = kpm.random_phases(m.n, 9, range(R))
    aug = np.concatenate([B, .5 * B[::-1]], axis=1)
    cfg = RunConfig(energy_eV=[0.], time_fs=[0., 1.], spectral_bounds=(-9.6, 9.6), axes=("x",))
    coeff, _ = kpm.bessel_coefficients(.5, cfg, weighted_tail=True)
    c, a = kpm.scaling(cfg)
    _, eng, _ = engine(m.H, m.S, precision=precision, velocity={"x": V})
    before = eng.lib.kmsd_kernel_launches()
    got = eng.series(aug, coeff, c, a, [[1., 0., 0.]])
    assert eng.lib.kmsd_kernel_launches() - before >= len(coeff) - 1
    want = O.engine_from_model(m.H, m.S, velocity={"x": V}).series(aug, coeff, c, a, [[1., 0., 0.]])
    assert_rel(got, want, TOL[precision], f"{velocity} {R}")
