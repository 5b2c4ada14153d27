"""Torch tensors whose values are not in memory as they read: lazily conjugated and
negated ones, transposes, slices and steps.  Each gives what its plain copy gives."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _views(torch, n, b, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    z = torch.randn((n, b), dtype=torch.complex128, device="cuda", generator=g)
    wide = torch.randn((n, 2 * b + 1), dtype=torch.complex128, device="cuda", generator=g)
    return {"conj": z.conj(), "mH": z.mT.contiguous().mH, "neg": torch._neg_view(z), "conj of neg": torch._neg_view(z).conj(),
            "transposed": z.mT.contiguous().mT, "slice": wide[:, 1:b + 1], "step": wide[:, ::2][:, :b],
            "conj slice": wide.conj()[:, 1:b + 1]}


@pytest.mark.parametrize("orthogonal", [True, False])
def test_views_equal_their_copies(cuda, orthogonal):
    import scipy.sparse as sp
    from tests.gpu_util import engine
    from tests.test_gpu_segmented import atom_model
    torch = cuda
    H, S, blocks = atom_model(66, 4)
    if orthogonal:
        S, blocks = sp.identity(H.shape[0], format="csr"), ()
    n = H.shape[0]
    velocity = {"x": (1j * (sp.triu(H, 1) - sp.tril(H, -1))).tocsr()}
    metric, eng, _ = engine(H, S, velocity=velocity, blocks=blocks)
    cfg = metric._create[2]
    for name, v in _views(torch, n, 4, 1).items():
        plain = v.resolve_conj().resolve_neg().clone(memory_format=torch.contiguous_format)
        cov = torch.randn((n, 3, 4), dtype=torch.complex128, device="cuda").conj()
        for call in (lambda x: eng.moments(x, 6, 0., 60.), lambda x: eng.h_action(x), lambda x: eng.v_cov([1., 0., 0.], x),
                     lambda x: eng.series(x, [1., .5j], 0., 60.), lambda x: eng.chain(x, 3, 0., 60.),
                     lambda x: metric.solve(x, cfg)[0], lambda x: eng.inner(x, x), lambda x: eng.H.matmul(x),
                     lambda x: eng.chain_correlate(x, cov, 3, 0., 60.),
                     lambda x: eng.chain_correlate(plain, x[:, None, :], 3, 0., 60.),
                     lambda x: torch.from_numpy(np.concatenate(eng.lanczos(x, 3)))):
            assert torch.equal(call(v), call(plain)), name
