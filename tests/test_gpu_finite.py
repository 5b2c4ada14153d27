"""The finiteness check of the inputs (kmsd_check_finite): every position of small
blocks and the edges of the kernel's passes, NaN and both infinities in either
part; the largest finite values pass."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _finite(torch, t):
    from kubomsd_b200 import _abi
    ok = C.c_int(-1)
    lib = _abi.require_library()
    assert lib.kmsd_check_finite(C.c_void_p(t.data_ptr()), t.numel(), C.byref(ok), None) == 0
    return ok.value


@pytest.mark.parametrize("count", [1, 3, 255, 257, 1025, 148 * 8 * 256 * 4, 148 * 8 * 256 * 4 + 5])
def test_check_finite(cuda, count):
    torch = cuda
    t = torch.full((count,), 1.7e308 - 1.7e308j, dtype=torch.complex128, device="cuda")
    torch.cuda.synchronize()
    assert _finite(torch, t) == 1
    at = range(count) if count < 4 else [0, 1, count // 2, 148 * 8 * 256 % count, count - 2, count - 1]
    for i in at:
        for bad in (complex(np.nan, 0), complex(0, np.nan), complex(np.inf, 1), complex(1, -np.inf)):
            t[i] = bad
            torch.cuda.synchronize()
            assert _finite(torch, t) == 0
        t[i] = 5e-324
    torch.cuda.synchronize()
    assert _finite(torch, t) == 1


def test_nonfinite_input_is_refused(cuda):
    import scipy.sparse as sp
    from kubomsd_b200.errors import NumericalError
    from tests.gpu_util import engine
    _, eng, _ = engine(sp.identity(40, format="csr"), sp.identity(40, format="csr"))
    B = np.ones((40, 2), complex)
    B[17, 1] = np.nan
    for call in (lambda: eng.moments(B, 4, 0., 2.), lambda: eng.h_action(B), lambda: eng.series(B, [1., 1.], 0., 2.),
                 lambda: eng.moments(cuda.from_numpy(B).cuda(), 4, 0., 2.)):
        with pytest.raises(NumericalError, match="expected finite"):
            call()
