"""One-launch metric solves beside one another and beside other kernels.

A solve's reductions run in a fixed order and its CTAs take their decisions from
the same bits, so a solve on a busy device returns exactly what it returns alone;
a value read before its writer published it would show as other bits, or as a
solve whose true residual misses its threshold."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# one cluster; the grid with the vectors in registers; the grid with the vectors in memory
@pytest.mark.parametrize("b", [8, 32, 64])
def test_solves_on_eight_streams_equal_solves_alone(cuda, b):
    from kubomsd_b200 import kpm, lattices
    from tests.gpu_util import engine
    torch = cuda
    m = lattices.diamond_sp3(cells=4, scale_hint=.24)  # 512 block rows, about 72 iterations
    S = m.S.tocsr()
    blocks = [(i, j, np.linalg.cholesky(S[i:j, i:j].toarray())) for i, j in m.atom_slices]
    metric, eng, _ = engine(m.H, S, blocks=blocks)
    cfg = metric._create[2]
    rng = np.random.default_rng(b)
    B = [torch.from_numpy(rng.standard_normal((S.shape[0], b)) + 1j * rng.standard_normal((S.shape[0], b))).cuda()
         for _ in range(8)]
    want = [metric.solve(x, cfg)[0].cpu() for x in B]
    replicas = [metric.replica() for _ in B]
    # steps of a large orthogonal lattice keep all SMs and the memory busy meanwhile
    hc = lattices.honeycomb(512, 256, seed=3, with_velocity=False)
    _, big, _ = engine(hc.H, hc.S, precision="mixed")
    psi = torch.from_numpy(kpm.random_phases(hc.n, 1, range(16))).cuda()
    big.moments(psi, 8, 0., 9.5)
    torch.cuda.synchronize()
    stop, errors, different = threading.Event(), [], []

    def load():
        with torch.cuda.stream(torch.cuda.Stream()):
            while not stop.is_set():
                big.moments(psi, 64, 0., 9.5)

    def work(i):
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                for _ in range(20):
                    if not torch.equal(replicas[i].solve(B[i], cfg)[0].cpu(), want[i]):
                        different.append(i)
        except Exception as exc:  # noqa: BLE001
            errors.append(exc)

    busy = threading.Thread(target=load)
    workers = [threading.Thread(target=work, args=(i,)) for i in range(8)]
    busy.start()
    for t in workers:
        t.start()
    for t in workers:
        t.join(timeout=300)
    stop.set()
    busy.join(timeout=60)
    assert not errors, errors
    assert not different, different
