"""Device memory of the RF simulation and the DTFT: what a call takes it gives
back, and it runs on any stream, with torch's memory or without."""
import numpy as np
import pytest

from conftest import gpu_available

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not gpu_available(), reason="needs a CUDA device")]


def _record(nt=200, n_rx=5, n_tx=3):
    g = np.random.default_rng(1)
    return np.arange(nt) * 1e-7, np.array([3e5, 5e5]), g.standard_normal((nt, n_rx, n_tx)), np.ones((n_tx, n_rx), bool)


def _simulate(tmp_path, n, n_tx, stream=None):
    from waveforminversionust_b200.simulate import wust_simulate
    model = dict(c_mps=np.full((n, n), 1500.0), x_m=np.arange(n) * .5e-3, y_m=np.arange(n) * .5e-3,
                 tx_index=np.arange(n_tx) * 3 + 1, rx_index=np.array([7, n * n - 3]), dt_s=60e-9,
                 source_pressure=np.array([0.0, 1.0, 0.5, 0.0]))
    cfg = dict(backend="native-batch", pml_size=20, density_kg_m3=1000, sound_speed_ref_mps=1550, downsample_factor=1,
               time_offset_s=0, work_dir=str(tmp_path))
    return wust_simulate(model, cfg, stream=stream)["pressure"]


def test_the_fields_of_a_large_simulation_go_back(tmp_path):
    """They are not left in torch's cache, where the library's own allocations cannot use them."""
    import torch
    from waveforminversionust_b200 import _lib
    need = _lib.load().wust_simulate_workspace_bytes(512, 512, 20, 64, 2, 4, 1, 0)
    assert need > 4 * _lib.WORKSPACE_LIMIT
    torch.cuda.empty_cache()
    reserved, free = torch.cuda.memory_reserved(), torch.cuda.mem_get_info()[0]
    _simulate(tmp_path, 512, 64)
    torch.cuda.synchronize()
    assert torch.cuda.memory_reserved() - reserved <= _lib.WORKSPACE_LIMIT
    assert free - torch.cuda.mem_get_info()[0] <= 2 * _lib.WORKSPACE_LIMIT      # and what the driver keeps for kernels


def test_streams_that_torch_does_not_know(tmp_path):
    """A stream is its handle: an object of the caller's own will do."""
    import torch
    from waveforminversionust_b200.prepare import dtft_device

    class Handle:
        def __init__(self, stream):
            self.cuda_stream, self.keep = stream.cuda_stream, stream

    own = Handle(torch.cuda.Stream())
    t, f, rf, active = _record()
    want = dtft_device(t, f, rf, active).cpu().numpy()
    rf = torch.as_tensor(rf, device="cuda")
    torch.cuda.synchronize()
    assert np.array_equal(dtft_device(t, f, rf, active, stream=own).cpu().numpy(), want)
    assert np.array_equal(_simulate(tmp_path, 24, 3, stream=own), _simulate(tmp_path, 24, 3))


def test_torch_without_memory(tmp_path, monkeypatch):
    import torch
    from waveforminversionust_b200.prepare import dtft_device
    record = _record()
    want = dtft_device(*record).cpu().numpy(), _simulate(tmp_path, 24, 3)
    empty = torch.empty

    def full(*a, **k):
        if k.get("dtype") == torch.uint8:
            raise torch.OutOfMemoryError("made up")
        return empty(*a, **k)

    monkeypatch.setattr(torch, "empty", full)
    assert np.array_equal(dtft_device(*record).cpu().numpy(), want[0])
    assert np.array_equal(_simulate(tmp_path, 24, 3), want[1])
