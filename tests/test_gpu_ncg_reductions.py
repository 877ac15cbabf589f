"""The NCG rules' reductions, finished by the last block on the device: one
block, blocks of one pass and of several, calls in a row and after a call that
failed.  Sums of n products in FP64, any order: n u |a||b| <= 2e5 * 1.1e-16 =
2.2e-11 relative to |a||b|, in practice sqrt(n) u; 1e-12 of |a||b|."""
import ctypes as C

import numpy as np
import pytest

from conftest import gpu_available

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not gpu_available(), reason="needs a CUDA device")]


@pytest.mark.parametrize("ny, nx", [(12, 14), (40, 47), (401, 400)])
def test_reductions_in_a_row_and_after_a_failure(ny, nx):
    import torch
    from waveforminversionust_b200 import _lib
    from waveforminversionust_b200._lib import WustError, check
    from waveforminversionust_b200.ncg import ncg_direction
    from waveforminversionust_b200.solver import HelmholtzSolver
    x, y = np.arange(nx) * 3e-4, np.arange(ny) * 3e-4
    s = HelmholtzSolver(x, y, np.full((ny, nx), 1500.0), None, 2e5, -1, 10.0, 3 * 3e-4,
                        dict(backend="gpu", stencil_bounds=(1400, 1700)))
    lib, h = _lib.load(), C.c_void_p(s.handle)
    rng = np.random.default_rng(nx)
    dev = lambda a: torch.as_tensor(np.ascontiguousarray(a.T), dtype=torch.float64, device="cuda")
    ptr = lambda t: C.c_void_p(t.data_ptr())
    for again in range(3):
        g, noise, prev, d = (rng.standard_normal((ny, nx)) for _ in range(4))
        z = g + 0.1 * noise
        gd, zd, pd, dd = dev(g), dev(z), dev(prev), dev(d)
        dot, beta, gz = C.c_double(), C.c_double(), C.c_double()
        check(lib.wust_ncg_dot(h, ptr(gd), ptr(dd), C.byref(dot)))
        assert abs(dot.value - np.sum(g * d)) <= 1e-12 * np.linalg.norm(g) * np.linalg.norm(d)
        check(lib.wust_ncg_direction(h, ptr(gd), ptr(zd), ptr(pd), 2.0 * g.size, 1, ptr(dd), C.byref(beta), C.byref(gz)))
        want, want_beta, want_gz = ncg_direction(g, z, prev, 2.0 * g.size, d, True)
        assert abs(gz.value - want_gz) <= 1e-12 * abs(want_gz) and abs(beta.value - want_beta) <= 1e-11
        assert np.abs(dd.cpu().numpy().T - want).max() <= 1e-10
        z[ny // 2, nx // 2] = np.nan                          # a failing call leaves the next one sound
        zd, dd = dev(z), dev(d)
        with pytest.raises(WustError, match="Invalid preconditioned gradient"):
            check(lib.wust_ncg_direction(h, ptr(gd), ptr(zd), ptr(pd), 1.0, 1, ptr(dd), C.byref(beta), C.byref(gz)))
    s.close()
