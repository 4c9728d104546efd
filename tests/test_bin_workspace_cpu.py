"""The binned forward's workspace: what the reconstruction server is charged
for it, and what a projection falls back to where memory is short."""

import numpy as np
import torch

import mbirtorch_b200 as mb
from mbirtorch_b200 import _lib, kernels
from mbirtorch_b200.serving import MemoryLedger

GIB = 1 << 30


def _cone512():
    m = mb.ConeBeamModel((720, 64, 768), np.linspace(0, 2 * np.pi, 720, endpoint=False),
                         source_detector_dist=4096.0, source_iso_dist=2048.0)
    m.set_params(no_warning=True, verbose=0, recon_shape=(512, 512, 32))
    return m


def test_ledger_charges_one_gib_of_records():
    """A 16-bit job holds its refresh's bins (FP32 jobs do not): 1 GiB of
    records for 512^2 pixels and 720 views, whose records in full are 7.7 GB."""
    m = _cone512()
    _, f32 = MemoryLedger.job_bytes(m, 'float32', False, 64)
    _, f16 = MemoryLedger.job_bytes(m, 'float16', False, 64)
    V, R, C = 720, 64, 768
    n = V * R * C
    # e in 16 bits, A delta in 16 bits, y in FP32 against e and A delta in FP32
    assert abs((f16 - f32) - (4 * n - 2 * n - 2 * n) - GIB) < 64 << 20


def test_larger_workspace_falls_back_to_the_default(monkeypatch):
    m = _cone512()
    g = m._geometry()
    pixels = int(mb.gen_full_indices((512, 512, 32)).size)
    sizes = {w: _lib.query('cpu', 'mbir_forward_project_binned_workspace_size_within', g, 720,
                           pixels, w) for w in (GIB, 2 * GIB)}
    assert sizes[GIB] == _lib.query('cpu', 'mbir_forward_project_binned_workspace_size', g, 720,
                                    pixels)
    assert GIB < sizes[2 * GIB] <= 2 * GIB + (1 << 20)
    proj = kernels.DeviceProjector(g, torch.zeros((720, 2)), torch.device('cpu'))
    asked = []

    def empty(n, dtype=None, device=None):
        asked.append(n)
        if n > GIB + (1 << 26):
            raise torch.OutOfMemoryError('no room')
        return n
    monkeypatch.setattr(kernels.torch, 'empty', empty)
    assert proj._binned_workspace('cpu', 720, pixels) == sizes[GIB]
    assert asked == [sizes[2 * GIB], sizes[GIB]]
    asked.clear()
    assert proj._binned_workspace('cpu', 720, pixels, lean=True) == sizes[GIB]
    assert asked == [sizes[GIB]]
