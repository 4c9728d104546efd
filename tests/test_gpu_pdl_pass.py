"""A partition pass launches each kernel behind the one before it while that
still runs (programmatic dependent launch); with per-launch timing on, each
waits for the whole of it.  Same bits: no kernel reads a cell before the
kernel that writes it has ended.  The sinograms' views and tiles are no
multiple of a 128-byte line, so that neighbouring tiles share lines, and the
subsets' bins come from the tail of the step before."""

import numpy as np
import pytest
import torch

import mbirtorch_b200 as mb
from mbirtorch_b200 import _lib
from mbirtorch_b200.vcd_engine import ResidentSinogram

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('kind', ['cone', 'parallel'])
@pytest.mark.parametrize('weighted', [False, True])
@pytest.mark.parametrize('code', [_lib.MBIR_F32, _lib.MBIR_F16])
def test_pass_equals_the_pass_with_ordinary_launches(kind, weighted, code):
    V, C, N = 90, 45, 30
    R, S = (44, 40) if kind == 'cone' else (36, 36)
    if kind == 'cone':
        m = mb.ConeBeamModel((V, R, C), np.linspace(0, 2 * np.pi, V, endpoint=False), 240.0, 120.0)
        m.set_params(no_warning=True, verbose=0, delta_det_channel=2.0, delta_det_row=2.0)
    else:
        m = mb.ParallelBeamModel((V, R, C), np.linspace(0, np.pi, V, endpoint=False))
        m.set_params(no_warning=True, verbose=0)
    m.auto_set_recon_geometry(no_warning=True)
    m.set_params(no_warning=True, recon_shape=(N, N, S), sigma_y=0.5, sigma_x=0.2)
    dev = torch.device('cuda', 0)
    gen = torch.Generator(device=dev).manual_seed(4)
    e0 = torch.randn((V, R, C), generator=gen, device=dev)
    w = torch.rand((V, R, C), generator=gen, device=dev) + 0.5 if weighted else None
    x0 = 0.1 * torch.rand((N * N, S), generator=gen, device=dev)
    H = m.compute_hessian_diagonal(weights=w, output_sharded=True).reshape(-1, S).contiguous()
    part = mb.gen_pixel_partition((N, N, S), 12, rng=np.random.RandomState(2))
    eng = m._make_engine(H, None if w is None else ResidentSinogram.from_vrc(w, code), code,
                         max_subset_pixels=part.shape[1])
    order = np.arange(part.shape[0], dtype=np.int32)
    out = []
    for timed in (True, False):
        flat, err = x0.clone(), ResidentSinogram.from_vrc(e0, code)
        acc = torch.zeros(2 + S, dtype=torch.float64, device=dev)
        torch.cuda.synchronize()
        before = _lib.timing_enable(timed)
        try:
            for _ in range(3):
                eng.partition_pass(flat, err, torch.as_tensor(part, device=dev), order, acc)
            torch.cuda.synchronize()
        finally:
            _lib.timing_enable(before)
            _lib.timing_collect()
        out.append((flat, err.data, acc))
    for a, b in zip(*out):
        assert torch.equal(a, b)
