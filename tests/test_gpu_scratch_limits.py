"""Calls on a device with little memory left: where the scratch of a one-launch path
does not fit, the call takes the path that needs less, as it did before there was
another.  The device is filled up to a stated rest, and given back."""
import ctypes as C
from contextlib import contextmanager

import pytest

pytestmark = pytest.mark.gpu


@contextmanager
def _left(torch, rest):
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    block = torch.empty(torch.cuda.mem_get_info()[0] - rest, dtype=torch.uint8, device="cuda")
    try:
        yield
    finally:
        torch.cuda.synchronize()
        del block
        torch.cuda.empty_cache()


@pytest.mark.parametrize("batch", [False, True])
def test_moments_without_room_for_the_cluster_sums(cuda, batch):
    """100,000 moments of 64 columns: the sums of the cluster path take 51 MB for
    each CTA of a cluster, the step kernels 8 MB of vectors."""
    from kubomsd_b200 import _abi, kpm, lattices
    from kubomsd_b200.batch import B200Batch
    from tests.gpu_util import engine
    torch = cuda
    M, b = 100_000, 64
    small, large = lattices.square_lattice(64, seed=1), lattices.square_lattice(180, seed=2)  # fits a cluster; does not
    B = torch.from_numpy(kpm.random_phases(small.n, 1, range(b))).cuda()
    wide = torch.from_numpy(kpm.random_phases(large.n, 1, range(b))).cuda()
    mu = torch.zeros((M, b), dtype=torch.float64, device="cuda")
    one = (C.c_double * 1)(0.), (C.c_double * 1)(12.)

    def make(m):
        if batch:
            return B200Batch([m.H], precision="fp64", tile_rows=64)
        return engine(m.H, m.S)[1]

    def run(obj, x, length):
        p, s = C.cast(C.c_void_p(mu.data_ptr()), C.POINTER(C.c_double)), C.c_void_p(torch.cuda.current_stream().cuda_stream)
        if batch:
            return obj.lib.kmsd_batch_moments(obj.handle, C.c_void_p(x.data_ptr()), p, b, length, *one,
                                              _abi.KMSD_MOMENTS_DOUBLING, 0, s)
        return obj.lib.kmsd_engine_moments(obj.handle, C.c_void_p(x.data_ptr()), p, b, length, 0., 12.,
                                           _abi.KMSD_MOMENTS_DOUBLING, s)

    warm, roomy, obj = make(large), make(small), make(small)
    assert run(warm, wide, 5) == 0  # the step kernels are loaded
    assert run(roomy, B, M) == 0
    want = mu.clone()
    assert run(obj, B, 5) == 0
    before = obj.lib.kmsd_kernel_launches()
    with _left(torch, 44 << 20):
        mu.zero_()
        rc = run(obj, B, M)
        got = mu.cpu()
    assert rc == 0, _abi.last_error(obj.lib)
    assert obj.lib.kmsd_kernel_launches() - before >= M // 2  # a launch per step
    assert float((got - want.cpu()).abs().max()) <= 1e-9 * float(want.abs().max())


def test_solve_without_room_for_padded_vectors(cuda):
    """33 columns run as 64 in one launch: seven vectors of 32,000 rows, 229 MB instead
    of 118.  The launch sequence solves them in what is left, on the same handle later
    too."""
    import numpy as np
    from kubomsd_b200 import lattices
    from tests.gpu_util import engine
    torch = cuda
    m = lattices.diamond_sp3(cells=10, scale_hint=.24)
    S = m.S.tocsr()
    blocks = [(i, j, np.linalg.cholesky(S[i:j, i:j].toarray())) for i, j in m.atom_slices]
    roomy, eng, _ = engine(m.H, S, blocks=blocks)
    cfg = roomy._create[2]
    tight, other = roomy.replica(), roomy.replica()
    B = torch.randn((S.shape[0], 33), dtype=torch.complex128, device="cuda")
    lib = roomy.lib

    def solve(metric):
        before = lib.kmsd_kernel_launches()
        x, report = metric.solve(B, cfg)
        assert report.converged.all()
        return x, lib.kmsd_kernel_launches() - before

    want, launches = solve(roomy)
    assert launches <= 3
    other.set_storage("mixed")
    solve(other)  # the kernels of the launch sequence are loaded
    torch.cuda.synchronize()
    with _left(torch, 190 << 20):
        got, launches = solve(tight)
        assert launches > 100
        again, _ = solve(tight)
        tight.solve(B[:, :4].contiguous(), cfg)
    # both meet |b - S x| <= 1e-10 |b|, kappa(S) is 50
    bound = 1.01 * 2 * 50 * 1e-10
    assert float(((got - want).norm(dim=0) / want.norm(dim=0)).max()) <= bound
    assert torch.equal(got, again)
