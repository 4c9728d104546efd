"""Detectors and cylinders large enough for the streamed cone forward and the
vector-column back projector, in the paths that other tests run on small ones:
several jobs' subset steps in one launch, and the refresh of the error
sinogram."""

import numpy as np
import pytest
import torch

import mbirtorch_b200 as mb
import test_gpu_batching as batching
from mbirtorch_b200 import _lib
from mbirtorch_b200._lib import ptr, stream_of
from mbirtorch_b200.vcd_engine import ResidentSinogram, partition_pass_batched

pytestmark = pytest.mark.gpu

DEV = torch.device('cuda', 0)


def _model(V, R, C, N, S, positivity=False):
    m = mb.ConeBeamModel((V, R, C), np.linspace(0, 2 * np.pi, V, endpoint=False),
                         12.0 * max(N, S), 6.0 * max(N, S))
    m.set_params(no_warning=True, verbose=0, delta_det_channel=2.0, delta_det_row=2.0)
    m.auto_set_recon_geometry(no_warning=True)
    m.set_params(no_warning=True, recon_shape=(N, N, S), positivity_flag=positivity)
    return m


@pytest.mark.parametrize('R,S,storage,weighted,positivity', [
    (200, 40, 'float32', False, False), (200, 200, 'float32', True, True),
    (208, 208, 'float16', True, False), (208, 70, 'bfloat16', False, True),
    (112, 100, 'float32', False, False),
])
def test_batched_pass_equals_each_jobs_own_pass(monkeypatch, R, S, storage, weighted, positivity):
    monkeypatch.setattr(batching, '_model', lambda kind, pos: _model(20, R, 40, 36, S, pos))
    jobs = [batching._job('cone', storage, weighted, positivity, 70 + j) for j in range(3)]
    single = []
    for eng, part, order, state in jobs:
        flat, err, acc = state()
        eng.partition_pass(flat, err, part, order, acc)
        single.append((flat, err, acc))
    states = [state() for _, _, _, state in jobs]
    partition_pass_batched([j[0] for j in jobs], [s[0] for s in states], [s[1] for s in states],
                           [j[1] for j in jobs], [j[2] for j in jobs], [s[2] for s in states])
    for (f1, e1, a1), (f2, e2, a2) in zip(single, states):
        assert bool(torch.isfinite(f1).all())
        assert torch.equal(f1, f2) and torch.equal(e1.data, e2.data) and torch.equal(a1, a2)


@pytest.mark.parametrize('R,S', [(200, 160), (320, 97), (200, 900)])
@pytest.mark.parametrize('storage', ['float32', 'float16'])
def test_error_refresh_binned_equals_scanning(R, S, storage):
    """e = (y - A x) / scale through the bins against the scanning forward.  A
    row's centre slice is formed in FP32 (S 2^-23), which is measured against
    ||y||; float16 adds one rounding of e."""
    m = _model(12, R, 56, 40, S)
    g = m._geometry()
    idx = torch.as_tensor(mb.gen_full_indices((40, 40, S)).astype(np.int64), device=DEV)
    flat = torch.rand(1600, S, device=DEV)
    y = m.projector.forward_volume(flat, idx)
    y += 0.1 * torch.randn_like(y)
    y_vcr = y.transpose(1, 2).contiguous()
    code = {'float32': _lib.MBIR_F32, 'float16': _lib.MBIR_F16}[storage]
    nb = int(_lib.query(DEV, 'mbir_forward_project_binned_workspace_size', g, g.num_views,
                        idx.shape[0]))
    outs = []
    for ws in (None, torch.empty(nb, dtype=torch.uint8, device=DEV)):
        err = ResidentSinogram.from_vrc(y, code)
        _lib.call(DEV, 'mbir_vcd_refresh_error', g, ptr(m.projector.view_params), ptr(flat),
                  ptr(idx), idx.shape[0], ptr(y_vcr), ptr(err.data), ptr(err.scale), code, ptr(ws),
                  0 if ws is None else ws.numel(), stream_of(DEV))
        outs.append(err.data.float() * err.scale.view(-1, 1, 1))
    d = float((outs[0] - outs[1]).norm() / y.norm())
    fp32 = max(1e-6, S * 2.0 ** -23)
    assert d <= fp32 + (0 if storage == 'float32' else
                        2.0 ** -10 * float(outs[0].norm() / y.norm()))
