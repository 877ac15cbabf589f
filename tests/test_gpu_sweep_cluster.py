"""The substitutions in one launch (a thread-block cluster takes its sources
through every column): each of the kernel's five tile shapes in both
directions against the FP64 substitution, on pages whose border nobody has
written, and the heights up to which a solve takes this path."""
import numpy as np
import pytest

from conftest import gpu_available

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not gpu_available(), reason="needs a CUDA device")]

NAMES = ("Ld", "Ll", "Lu", "Dd", "Dl", "Du", "Ud", "Ul", "Uu")


def _operator(ny, nx, pml=2, dx=0.4e-3, f=0.6e6):
    x, y = (np.arange(nx) - (nx - 1) / 2) * dx, (np.arange(ny) - (ny - 1) / 2) * dx
    c = 1500 + 20 * np.random.default_rng(ny * 1000 + nx).standard_normal((ny, nx))
    return x, y, c, f, pml * dx


# (rows, sources) whose plan is the shape of 16 x 2, 32 x 4, 48 x 8, 64 x 8 (at even and odd heights: a page column's
# first byte, and K in whole stages or not) and 96 x 12, there with the ring of two stages (H) and of three (H^H)
@pytest.mark.parametrize("ny, S", [(34, 3), (64, 6), (65, 9), (224, 32), (131, 256), (132, 250), (230, 256), (331, 128),
                                   (401, 20), (402, 20), (552, 30), (553, 30), (570, 13)])
@pytest.mark.parametrize("adjoint", [False, True])
def test_every_shape_matches_the_fp64_substitution(ny, S, adjoint):
    import torch
    from oracle import helmholtz_fp64 as o
    from waveforminversionust_b200.solver import applyBlockLU, decompBlockLU
    nx = 4
    x, y, c, f, L = _operator(ny, nx)
    coefs = o.HelmholtzSolverFP64(x, y, c, np.zeros((ny, nx)), f, -1, 10.0, L,
                                  dict(backend="cpu", stencil_bounds=(1400, 1700)), factor=False).coefs
    dev = [torch.as_tensor(np.ascontiguousarray(coefs[n].astype(np.complex64).T), device="cuda").t() for n in NAMES]
    inv = decompBlockLU(*dev)
    pages = inv.cpu().numpy().astype(np.complex128)
    # the substitution is that of the interior rows and columns: what stands around them is not read
    for edge in (inv[0], inv[-1], inv[:, 0], inv[:, -1]):
        edge.fill_(complex(np.nan, np.inf))
    g = np.random.default_rng(S)
    src = (g.standard_normal((ny, nx, S)) + 1j * g.standard_normal((ny, nx, S))).astype(np.complex64)
    u = applyBlockLU(src, *[dev[i] for i in (0, 1, 2, 6, 7, 8)], inv, adjoint).cpu().numpy()
    want = o.block_lu_apply(src.astype(np.complex128), {n: coefs[n].astype(np.complex64) for n in NAMES}, pages, adjoint)
    # 2 (nx - 1) products of n terms in 32 bits, rounded like a random walk: 2e-5 leaves an order of magnitude
    assert np.linalg.norm(u - want) < 2e-5 * np.linalg.norm(want)


# the widest tile with two stages of the ring fits up to 570 rows (H) and 642 (H^H)
@pytest.mark.parametrize("ny, adjoint, one", [(64, False, True), (64, True, True), (552, False, True), (570, False, True),
                                              (571, False, False), (571, True, True), (642, True, True), (643, True, False)])
def test_heights_that_take_one_launch(ny, adjoint, one):
    from oracle import helmholtz_fp64 as o
    from waveforminversionust_b200.solver import HelmholtzSolver
    nx, S = 24, 5
    x, y, c, f, L = _operator(ny, nx)
    s = HelmholtzSolver(x, y, c, None, f, -1, 10.0, L, dict(backend="gpu", stencil_bounds=(1400, 1700)), precision="c64",
                        max_sources=S)
    try:
        g = np.random.default_rng(ny)
        src = np.zeros((ny, nx, S), np.complex64)
        src[1:-1, 1:-1] = (g.standard_normal((ny - 2, nx - 2, S)) + 1j * g.standard_normal((ny - 2, nx - 2, S)))
        u = s.solve(src, adjoint=adjoint).cpu().numpy()
        launches = s.stats()["kernel_launches"]            # of the solve
        assert launches < nx if one else launches >= 4 * (nx - 1)
        coefs = {n: getattr(s, n).cpu().numpy().astype(np.complex128) for n in ("Ld", "Ll", "Lu", "Ud", "Ul", "Uu")}
        want = o.block_lu_apply(src.astype(np.complex128), coefs, s.invT.cpu().numpy().astype(np.complex128), adjoint)
        assert np.linalg.norm(u - want) < 2e-5 * np.linalg.norm(want)
    finally:
        s.close()


# caps that hold all of a solve's clusters (the first two) and 9 of 16, 10 of 25, 4 of 8, 3 of 6, 1 of 8, 1 of 3: so many
# launches, each of no more CTAs than the cap
@pytest.mark.parametrize("ny, S, cap, launches", [(224, 32, 37, 1), (64, 7, 3, 1), (224, 128, 37, 2), (130, 200, 20, 3),
                                                  (300, 64, 37, 2), (552, 64, 20, 2), (130, 64, 3, 8), (34, 32, 1, 3)])
@pytest.mark.parametrize("adjoint", [False, True])
def test_a_cap_on_the_ctas_is_kept(ny, S, cap, launches, adjoint):
    from oracle import helmholtz_fp64 as o
    from waveforminversionust_b200.solver import HelmholtzSolver
    nx = 12
    x, y, c, f, L = _operator(ny, nx)
    g = np.random.default_rng(ny)
    src = np.zeros((ny, nx, S), np.complex64)
    src[1:-1, 1:-1] = g.standard_normal((ny - 2, nx - 2, S)) + 1j * g.standard_normal((ny - 2, nx - 2, S))
    count = {}
    for max_ctas in (0, cap):
        s = HelmholtzSolver(x, y, c, None, f, -1, 10.0, L, dict(backend="gpu", stencil_bounds=(1400, 1700)), precision="c64",
                            max_sources=S, max_ctas=max_ctas)
        try:
            u = s.solve(src, adjoint=adjoint).cpu().numpy()
            count[max_ctas] = s.stats()["kernel_launches"]
            coefs = {n: getattr(s, n).cpu().numpy().astype(np.complex128) for n in ("Ld", "Ll", "Lu", "Ud", "Ul", "Uu")}
            want = o.block_lu_apply(src.astype(np.complex128), coefs, s.invT.cpu().numpy().astype(np.complex128), adjoint)
            assert np.linalg.norm(u - want) < 2e-5 * np.linalg.norm(want)
        finally:
            s.close()
    assert count[0] < nx and count[cap] == count[0] + launches - 1, count
