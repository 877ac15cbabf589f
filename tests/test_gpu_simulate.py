"""The RF simulation's paths against the FP64 oracle, at the sizes where a
split or a transform plan can go wrong.

Tolerance: the fields are FP32 (unit roundoff u = 6e-8) through four
transforms a step of up to 12 log2(n) rounding steps each, errors of the steps
adding up at worst in proportion to their number: u * 4 * 12 * 40 = 1.2e-4
relative for 40 steps; 1e-4 is what the pipeline case above holds in 400."""
import numpy as np
import pytest

from conftest import gpu_available

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not gpu_available(), reason="needs a CUDA device")]


@pytest.mark.parametrize("ny, nx, pml, n_tx, tx_batch, q, own", [
    (2, 3, 1, 2, 0, 1, True),              # 4 x 5: blocks of a cluster without rows or columns
    (11, 9, 2, 3, 0, 1, True),             # 15 x 13
    (23, 27, 10, 3, 0, 2, True),           # 43 x 47, both prime
    (40, 44, 10, 40, 0, 1, True),          # 60 x 64, more transmitters than widest clusters fit
    (40, 43, 10, 5, 2, 3, True),           # 60 x 63 (7), a last batch of one
    (93, 89, 10, 2, 0, 1, True),           # 113 x 109, the largest primes of a cluster
    (108, 118, 10, 2, 0, 1, True),         # 128 x 138 (23 by direct sums)
    (220, 222, 10, 3, 2, 2, True),         # 240 x 242: tiles, 11 11 2
    (239, 246, 10, 2, 0, 1, True),         # 259 x 266 (37, 19)
    (253, 301, 10, 2, 0, 1, False),        # 273 x 321 (107): a prime beyond the tiles' rule, library transforms
    (172, 880, 10, 2, 0, 1, True),        # 192 x 900: x tiles of four columns
    (104, 125, 12, 3, 2, 2, False),        # 128 x 149: library transforms
])
def test_simulation_matches_the_oracle(tmp_path, ny, nx, pml, n_tx, tx_batch, q, own):
    from oracle import kwave_fp64 as k
    from waveforminversionust_b200 import _lib
    from waveforminversionust_b200.simulate import wust_simulate
    rng = np.random.default_rng(ny * 1000 + nx)
    d, dt, nt = .5e-3, 60e-9, 40
    c = 1500 + 40 * rng.random((ny, nx))
    at = rng.permutation(ny * nx) + 1
    tx = at[:n_tx]
    rx = np.concatenate([tx[:1], at[::-1][:min(6, ny * nx - 1)]])            # one on a source, the others anywhere
    rx = np.unique(rx)[::-1]
    t = np.arange(nt) * dt
    src = np.sin(2 * np.pi * .8e6 * t) * np.exp(-((t - 1e-6) / 5e-7) ** 2)
    model = dict(c_mps=c, x_m=np.arange(nx) * d, y_m=np.arange(ny) * d, tx_index=tx, rx_index=rx, dt_s=dt, source_pressure=src)
    cfg = dict(backend="native-batch", pml_size=pml, density_kg_m3=1000, sound_speed_ref_mps=1550, downsample_factor=q,
               time_offset_s=0, work_dir=str(tmp_path), tx_batch=tx_batch)
    assert (_lib.load().wust_simulate_workspace_bytes(ny, nx, pml, n_tx, rx.size, nt, q, tx_batch) > 0) == own
    got = wust_simulate(model, cfg)["pressure"]
    ref = k.simulate(c, d, d, dt, src, tx, rx, pml, 1550, 1000)             # [rx, tx, time]
    if q > 1:
        ref = k.decimate(ref, q)
    want = np.transpose(ref, (2, 0, 1))
    assert got.shape == want.shape
    assert np.linalg.norm(got - want) < 1.2e-4 * np.linalg.norm(want)


def test_threads_with_grids_of_different_sizes(tmp_path):
    """Calls from several threads, each with a grid of its own, give what they
    give one after another."""
    import threading
    import torch
    from waveforminversionust_b200.simulate import wust_simulate
    t = np.arange(12) * 60e-9
    src = np.sin(2 * np.pi * .8e6 * t)

    def call(ny, nx, stream):
        model = dict(c_mps=np.full((ny, nx), 1500.0), x_m=np.arange(nx) * .5e-3, y_m=np.arange(ny) * .5e-3,
                     tx_index=np.array([5, 9]), rx_index=np.array([ny * nx - 3]), dt_s=60e-9, source_pressure=src)
        cfg = dict(backend="native-batch", pml_size=6, density_kg_m3=1000, sound_speed_ref_mps=1550, downsample_factor=1,
                   time_offset_s=0, work_dir=str(tmp_path))
        return wust_simulate(model, cfg, stream=stream)["pressure"]

    sizes = [(12, 14), (100, 116), (228, 244), (52, 54), (180, 276)]
    want = [call(*s, None) for s in sizes]
    wrong = []

    def run(k):
        stream = torch.cuda.Stream()
        for _ in range(6):
            try:
                if not np.array_equal(call(*sizes[k], stream), want[k]):
                    wrong.append((sizes[k], "differs"))
            except Exception as e:                                        # noqa: BLE001
                wrong.append((sizes[k], e))
    threads = [threading.Thread(target=run, args=(k,)) for k in range(len(sizes))]
    for th in threads:
        th.start()
    for th in threads:
        th.join()
    assert not wrong
