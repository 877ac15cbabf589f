"""Complex-single block LU at the sizes where its kernels change shape: the
factorization against the FP64 recursion at the edges of its tiles, pivot
blocks and of the dataflow kernel's range, and its report of singular pages."""
import numpy as np
import pytest

from conftest import gpu_available

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not gpu_available(), reason="needs a CUDA device")]

NAMES = ("Ld", "Ll", "Lu", "Dd", "Dl", "Du", "Ud", "Ul", "Uu")


def _blocks(ny, nx, pml=2, dx=0.4e-3, f=0.6e6):
    from oracle import helmholtz_fp64 as o
    x, y = (np.arange(nx) - (nx - 1) / 2) * dx, (np.arange(ny) - (ny - 1) / 2) * dx
    rng = np.random.default_rng(ny * 1000 + nx)
    c = 1500 + 20 * rng.standard_normal((ny, nx))
    s = o.HelmholtzSolverFP64(x, y, c, np.zeros((ny, nx)), f, -1, 10.0, pml * dx,
                              dict(backend="cpu", stencil_bounds=(1400, 1700)), factor=False)
    return s.coefs


def _device(coefs):
    import torch
    return [torch.as_tensor(np.ascontiguousarray(coefs[n].astype(np.complex64).T), device="cuda").t() for n in NAMES]


# interior rows 1, a pivot block and one more, a tile and one more, two tiles less one, the largest page of one tile
# per CTA, and the first page beyond it
@pytest.mark.parametrize("ny,nx", [(3, 5), (18, 7), (19, 7), (50, 6), (51, 6), (97, 5), (146, 9), (578, 4), (579, 4)])
def test_factor_matches_the_fp64_recursion(ny, nx):
    from oracle import helmholtz_fp64 as o
    from waveforminversionust_b200.solver import decompBlockLU
    coefs = _blocks(ny, nx)
    got = decompBlockLU(*_device(coefs)).cpu().numpy()
    want = o.block_lu_factor({n: coefs[n].astype(np.complex64).astype(np.complex128) for n in NAMES})
    assert got.shape == want.shape
    for j in range(nx):                                   # page by page: the Dirichlet columns are identities
        assert np.linalg.norm(got[:, :, j] - want[:, :, j]) < 2e-5 * np.linalg.norm(want[:, :, j]), j
    assert not got[[0, -1]].any() and not got[:, [0, -1]].any()


@pytest.mark.parametrize("ny,row", [(20, 1), (20, 2), (60, 17), (60, 50)])
def test_factor_reports_a_singular_page(ny, row):
    """A row of zeros in one page: the page is named, and the next call works."""
    from waveforminversionust_b200._lib import WustError
    from waveforminversionust_b200.solver import decompBlockLU
    coefs = {n: v.copy() for n, v in _blocks(ny, 6).items()}
    good = decompBlockLU(*_device(coefs)).cpu().numpy()
    bad = {n: v.copy() for n, v in coefs.items()}
    bad["Dd"][row, 0] = 0                                  # the first page is the identity: decoupled rows
    with pytest.raises(WustError, match=rf"block 1 is singular at pivot {row}"):
        decompBlockLU(*_device(bad))
    assert np.array_equal(decompBlockLU(*_device(coefs)).cpu().numpy(), good)


# one interior row; odd and even column lengths (the parity of a page column's first byte); columns that take a launch
# per column step (H beyond 570 rows, H^H beyond 642; the shapes of the one launch are in test_gpu_sweep_cluster.py)
@pytest.mark.parametrize("ny,nx,S", [(3, 3, 1), (3, 5, 3), (18, 7, 5), (19, 6, 2), (64, 9, 13), (97, 8, 1), (194, 5, 40),
                                     (195, 5, 41), (578, 4, 30), (642, 4, 20), (770, 4, 3), (771, 4, 3)])
@pytest.mark.parametrize("adjoint", [False, True])
def test_sweeps_match_the_fp64_substitution(ny, nx, S, adjoint):
    """The substitutions on given pages, sources on the border included, from views on 16 and on 8 bytes."""
    import torch
    from oracle import helmholtz_fp64 as o
    from waveforminversionust_b200.solver import applyBlockLU, decompBlockLU
    coefs = _blocks(ny, nx)
    dev = _device(coefs)
    inv = decompBlockLU(*dev)
    g = np.random.default_rng(S)
    src = (g.standard_normal((ny, nx, S)) + 1j * g.standard_normal((ny, nx, S))).astype(np.complex64)
    sides = [dev[i] for i in (0, 1, 2, 6, 7, 8)]
    u = applyBlockLU(src, *sides, inv, adjoint).cpu().numpy()
    want = o.block_lu_apply(src.astype(np.complex128), {n: coefs[n].astype(np.complex64) for n in NAMES},
                            inv.cpu().numpy().astype(np.complex128), adjoint)
    # 2 (nx - 1) products of n terms in 32 bits, rounded like a random walk: 2e-5 leaves an order of magnitude
    assert np.linalg.norm(u - want) < 2e-5 * np.linalg.norm(want)
    shifted = torch.empty(nx * ny * ny + 1, dtype=torch.complex64, device="cuda")[1:].view(nx, ny, ny)
    shifted.copy_(inv.permute(2, 1, 0))
    v = applyBlockLU(src, *sides, shifted.permute(2, 1, 0), adjoint).cpu().numpy()
    assert np.linalg.norm(v - want) < 2e-5 * np.linalg.norm(want)
