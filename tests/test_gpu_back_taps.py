"""Back projectors that leave out the channel taps of zero weight: the same
bits as with every tap read, and infinities and NaNs reach the same voxels.
The layout change looks for those only where the kernel reads the answer, and
takes no workspace from the partial sums."""

import numpy as np
import pytest
import torch

import oracle
from conftest import rel_l2
from mbirtorch_b200 import _lib, kernels
from oracle import OracleGeometry

pytestmark = pytest.mark.gpu


def _projector(kind, V, R, C, N, S, pitch):
    ang = np.linspace(0, np.pi, V, endpoint=False)
    vp = np.stack([ang, np.zeros(V)], axis=1).astype(np.float32)
    if kind == 'parallel':
        g = kernels.make_geometry('parallel', V, R, C, N, N, S, 1, delta_det_channel=pitch,
                                  det_channel_offset=0.3)
    else:
        g = kernels.make_geometry('cone', V, R, C, N, N, S, 1, 1, False, 2.0 * pitch, 2.0, 0.3, 0.0,
                                  1.0, 1.0, 1.0, 0.0, 2.0, 8.0 * N)
    return kernels.DeviceProjector(g, vp, torch.device('cuda', 0)), vp


@pytest.mark.parametrize('kind', ['parallel', 'cone'])
@pytest.mark.parametrize('pitch', [1.0, 0.72])   # footprints of two cells; of two or three
@pytest.mark.parametrize('bad', [None, float('inf'), float('nan')])
def test_zero_taps_left_out(kind, pitch, bad):
    """Parallel beam leaves them out from 96 M voxel-views on; cone beam reads
    every tap in either layout, and checks the layouts against each other."""
    V, R, C, N = 66, 128, 520, 112
    assert N * N * V * R >= 96e6
    proj, _ = _projector(kind, V, R, C, N, R, pitch)
    gen = torch.Generator(device='cuda').manual_seed(3)
    y = torch.randn((V, R, C), generator=gen, device='cuda')
    idx = torch.arange(N * N, device='cuda')
    if bad is not None:
        y[5, 60:70, C // 2 - 3] = bad
    for power in (1, 2):
        skip = proj.back(y, idx, coeff_power=power)               # scanned by the layout change
        every = proj.back(y.transpose(1, 2).contiguous(), idx, coeff_power=power,
                          layout=_lib.MBIR_LAYOUT_VCR)            # reads every tap
        assert torch.equal(torch.isnan(skip), torch.isnan(every))
        assert torch.equal(torch.nan_to_num(skip), torch.nan_to_num(every))
        assert bool(torch.isfinite(skip).all()) == (bad is None)


def _back_into(proj, y, idx, band, ws, ws_bytes):
    out = torch.empty((idx.numel(), band), device='cuda')
    _lib.call(y.device, 'mbir_back_project', proj.geom, _lib.ptr(proj.view_params), 0, y.shape[0],
              _lib.ptr(y), _lib.MBIR_LAYOUT_VRC, _lib.ptr(idx), idx.numel(), 1, 0, band,
              _lib.ptr(out), _lib.ptr(ws), ws_bytes, _lib.stream_of(y.device))
    return out


@pytest.mark.parametrize('kind,N', [('cone', 60), ('parallel', 60)])
def test_nothing_scans_where_no_tap_is_left_out(kind, N):
    """Cone beam, and parallel beam too small to gain: the workspace behind the
    layout change and the partials is not written (a flag would be)."""
    V, R, C = 66, 128, 520                      # 4.4 M cells
    proj, _ = _projector(kind, V, R, C, N, R, 1.0)
    idx = torch.arange(N * N, device='cuda')
    y = torch.rand((V, R, C), device='cuda')
    size = int(_lib.query(y.device, 'mbir_back_project_workspace_size', proj.geom, V, idx.numel(),
                          R))
    ws = torch.full((size + 4096,), 0xAB, dtype=torch.uint8, device='cuda')
    got = _back_into(proj, y, idx, R, ws, size + 4096)
    assert torch.equal(got, proj.back(y, idx))
    used = V * R * C * 4
    part = idx.numel() * R * 4
    while used + part <= size:                  # whole partial volumes
        used += part
    assert bool((ws[used:] == 0xAB).all())


@pytest.mark.parametrize('N', [60, 112])        # without and with the scan
def test_flag_takes_nothing_from_the_partials(N):
    """The smallest workspace for all view chunks gives the default's bits."""
    V, R, C = 66, 128, 520
    proj, _ = _projector('parallel', V, R, C, N, R, 1.0)
    idx = torch.arange(0, N * N, 7 if N == 60 else 1, device='cuda')
    y = torch.rand((V, R, C), device='cuda')
    sino, part = V * R * C * 4, idx.numel() * R * 4
    size = int(_lib.query(y.device, 'mbir_back_project_workspace_size', proj.geom, V, idx.numel(),
                          R))
    chunks = (size - sino) // part
    assert chunks > 1 or N == 112
    exact = sino + chunks * part
    ws = torch.empty(size, dtype=torch.uint8, device='cuda')
    assert torch.equal(_back_into(proj, y, idx, R, ws, exact), proj.back(y, idx))


def test_workspace_without_room_for_the_flag():
    """A workspace that holds the layout change alone still serves."""
    V, R, C, N = 66, 128, 520, 8
    proj, _ = _projector('parallel', V, R, C, N, R, 1.0)
    y = torch.rand((V, R, C), device='cuda')
    idx = torch.arange(N * N, device='cuda')
    want = proj.back(y, idx)
    out = torch.empty_like(want)
    ws = torch.empty(V * R * C * 4, dtype=torch.uint8, device='cuda')
    _lib.call(y.device, 'mbir_back_project', proj.geom, _lib.ptr(proj.view_params), 0, V,
              _lib.ptr(y), _lib.MBIR_LAYOUT_VRC, _lib.ptr(idx), idx.numel(), 1, 0, R,
              _lib.ptr(out), _lib.ptr(ws), ws.numel(), _lib.stream_of(y.device))
    # one view chunk instead of several: another order of FP32 sums
    assert rel_l2(out.cpu().numpy(), want.cpu().numpy()) <= 1e-6


@pytest.mark.parametrize('rows', [12, 16, 20, 64, 68, 128, 132, 260])
@pytest.mark.parametrize('pitch', [1.0, 0.72])
def test_parallel_back_matches_oracle(rows, pitch):
    V, C, N = 45, 37, 19
    proj, vp = _projector('parallel', V, rows, C, N, rows, pitch)
    og = OracleGeometry(num_det_rows=rows, num_det_channels=C, num_recon_rows=N, num_recon_cols=N,
                        num_slices=rows, delta_det_channel=pitch, det_channel_offset=0.3,
                        psf_radius=1)
    rng = np.random.default_rng(rows)
    idx = np.sort(rng.choice(N * N, size=101, replace=False)).astype(np.int64)
    y = rng.standard_normal((V, rows, C)).astype(np.float32)
    for power in (1, 2):
        got = proj.back(torch.as_tensor(y).cuda(), torch.as_tensor(idx).cuda(), coeff_power=power)
        want = oracle.parallel_back(og, vp[:, 0].astype(np.float64), y, idx, power)
        assert rel_l2(got.cpu().numpy(), want) <= 1e-5
