"""The GPU DTFT at the sizes where its kernels change shape: odd and even
records, ragged tails of the pair blocks, frequency octets and passes, warps
that split a trace's samples or not, both types, aligned and not, and the two
routes (evenly spaced samples, others) against each other and FP64."""
import numpy as np
import pytest

from conftest import gpu_available

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not gpu_available(), reason="needs a CUDA device")]

DT = 1 / 12.5e6


def _record(nt, n_rx, n_tx, nf, dtype, shift=0.0):
    g = np.random.default_rng(nt + 7 * n_rx + 31 * nf)
    t = -3e-6 + np.arange(nt) * DT
    if shift:                                             # off the even grid, inside the accepted 1e-6 of a step
        t = t + shift * DT * g.uniform(-1, 1, nt)
    f = g.permutation(np.linspace(0.02, 0.49, nf)) / DT
    return t, f, g.standard_normal((nt, n_rx, n_tx)).astype(dtype), g.random((n_tx, n_rx)) > 0.1


def _want(t, f, p, active):
    k = np.exp(-2j * np.pi * f[:, None] * t[None]) * (t[1] - t[0])
    y = np.einsum("kt,trx->xrk", k, p.astype(np.float64))
    return y * active[:, :, None]


@pytest.mark.parametrize("nt,n_rx,n_tx,nf", [(2, 1, 1, 1), (3, 2, 1, 1), (16, 3, 2, 8), (31, 9, 5, 9), (32, 8, 1, 16), (33, 1, 8, 17),
                                             (256, 5, 3, 40), (257, 4, 4, 41), (130, 3, 2, 300), (264, 70, 64, 11),
                                             (72, 150, 130, 3)])
@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("shift", [0.0, 2e-7])
def test_dtft_matches_fp64(nt, n_rx, n_tx, nf, dtype, shift):
    """Both routes, to the rounding of the complex single result (2^-24 per
    component); a nonfinite sample counts on active channels only."""
    import torch
    from waveforminversionust_b200._lib import WustError
    from waveforminversionust_b200.prepare import dtft_device
    t, f, p, active = _record(nt, n_rx, n_tx, nf, dtype, shift)
    active[0, 0] = True
    want = _want(t, f, p, active)
    got = dtft_device(t, f, p, active).cpu().numpy()
    assert got.shape == want.shape and not got[~active].any()
    assert np.linalg.norm(got - want) < 2 ** -23 * np.linalg.norm(want)
    # the same samples one element off any 16-byte boundary
    raw = torch.empty(nt * n_rx * n_tx + 1, dtype=torch.as_tensor(p).dtype, device="cuda")[1:].view(n_tx, n_rx, nt)
    raw.copy_(torch.as_tensor(np.ascontiguousarray(p.transpose(2, 1, 0))))
    assert np.array_equal(dtft_device(t, f, raw.permute(2, 1, 0), active).cpu().numpy(), got)
    for value in (np.nan, np.inf):
        q = p.copy()
        q[nt // 2, 0, 0] = value
        with pytest.raises(WustError, match="Nonfinite RF on an active channel"):
            dtft_device(t, f, q, active)
        if not active.all():
            x, r = np.argwhere(~active)[0]
            q = p.copy()
            q[-1, r, x] = value
            assert np.array_equal(dtft_device(t, f, q, active).cpu().numpy(), got)
