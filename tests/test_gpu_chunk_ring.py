"""The chunked sweeps at the sizes where their operand ring changes its shape
(chunks per stage by the number of sources, steps of fewer chunks than the
ring has stages, a last stage that is not full) and where a tile's rows end:
against the sequential sweeps, both refined to 1e-9.

Tolerance: the fields are rounded to complex single (6e-8) from iterates
within 1e-9 of the same solution: 2e-9 + 2 * 6e-8 / sqrt(3) < 1e-7."""
import numpy as np
import pytest

from conftest import gpu_available

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not gpu_available(), reason="needs a CUDA device")]


@pytest.mark.parametrize("ny, nx, S", [(18, 40, 5), (66, 41, 16), (67, 40, 64), (130, 33, 65), (131, 50, 128), (228, 45, 129),
                                       (196, 36, 200), (290, 34, 256)])
def test_chunked_sweeps_at_the_edges_of_the_ring(ny, nx, S):
    from waveforminversionust_b200.solver import HelmholtzSolver
    dx = 0.3e-3
    x = (np.arange(nx) - (nx - 1) / 2) * dx
    y = (np.arange(ny) - (ny - 1) / 2) * dx
    X, Y = np.meshgrid(x, y)
    c = 1500 + 40 * np.exp(-((X - 1e-3) ** 2 + Y ** 2) / (2 * (4e-3) ** 2))
    g = np.random.default_rng(ny + S)
    r = np.zeros((ny, nx, S), np.complex64)
    r[1:-1, 1:-1] = g.standard_normal((ny - 2, nx - 2, S)) + 1j * g.standard_normal((ny - 2, nx - 2, S))
    sols = {}
    for method, correction in (("default", "default"), ("default", "same"), ("sequential", "same")):
        s = HelmholtzSolver(x, y, c, None, 0.8e6, -1, 10.0, 4 * dx, dict(backend="gpu", stencil_bounds=(1400, 1700)),
                            precision="tf32-refined", refine_tol=1e-9, max_sources=S, sweep_method=method,
                            correction_precision=correction)
        for adjoint in (False, True):
            sols[method, correction, adjoint] = s.solve(r, adjoint=adjoint).detach().cpu().numpy()[1:-1, 1:-1]
            assert s.stats()["error_estimate"] <= 1e-9
        s.close()
    for adjoint in (False, True):
        want = sols["sequential", "same", adjoint]
        for correction in ("default", "same"):
            got = sols["default", correction, adjoint]
            assert np.linalg.norm(got - want) < 1e-7 * np.linalg.norm(want), correction
