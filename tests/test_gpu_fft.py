"""FFT endpoints vs numpy FFTs (marked gpu).

Gates from the reference's custom-FFT self checks (nufft_integrated_bench.cu:1217-1237,
:1264-1280): forward panel rel_l2 <= 5e-4, inverse rel_l2 <= 2e-5.  The FP16 high +
residual panel carries ~2^-22 relative precision, so the forward is held to 1e-5 here.
"""
import numpy as np
import pytest

from gpu_cases import case, rel_l2
from oracle import kb as okb

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def _grid_from_image(img, g, shift):
    """[C, G, G] padded grid: position n holds image index (n + shift) mod G (if < N)."""
    c, n, _ = img.shape
    out = np.zeros((c, g, g), dtype=np.complex128)
    pos = (np.arange(n) - shift) % g
    out[:, pos[:, None], pos[None, :]] = img
    return out


@pytest.mark.parametrize("name,layout", [("small", "centered"), ("small", "reference"), ("cfg0", "centered"),
                                         ("headline", "centered"), ("c16", "reference"), ("n192", "centered"),
                                         ("n320", "reference")])
def test_forward_panel_matches_numpy_fft(name, layout):
    from trajsparsenufft_b200.operator import Plan
    traj, x, s, n, g, c, j, _ = case(name)
    plan = Plan.from_trajectory(traj, im_size=n, grid_size=g, coils=c, width=j,
                                reference_layout=(layout == "reference"))
    panel, scale = plan.fft_forward_panel(torch.from_numpy(x).cuda(), torch.from_numpy(s).cuda())
    p = panel.float().cpu().numpy().astype(np.float64)            # [G*G, 4C], rows q1*G + q0
    hi, res = p[:, : 2 * c], p[:, 2 * c:]
    v = (hi + res)[:, 0::2] + 1j * (hi + res)[:, 1::2]            # [G*G, C]
    got = v.reshape(g, g, c).transpose(2, 1, 0) / scale           # [C, q0, q1]
    d = okb.deapodization(n, g, j)
    shift = 0 if layout == "reference" else n // 2
    want = np.fft.fft2(_grid_from_image(x[None] * s * d[None], g, shift))
    assert rel_l2(got, want) <= 1e-5


@pytest.mark.parametrize("name,layout", [("small", "centered"), ("cfg0", "reference"), ("headline", "centered"),
                                         ("c16", "centered"), ("n192", "reference"), ("n320", "centered")])
def test_adjoint_endpoint_matches_numpy_ifft(name, layout):
    from trajsparsenufft_b200.operator import Plan
    traj, x, s, n, g, c, j, _ = case(name)
    plan = Plan.from_trajectory(traj, im_size=n, grid_size=g, coils=c, width=j,
                                reference_layout=(layout == "reference"))
    rng = np.random.default_rng(5)
    grid = (rng.standard_normal((c, g, g)) + 1j * rng.standard_normal((c, g, g))).astype(np.complex64)
    internal = np.ascontiguousarray(grid.transpose(2, 1, 0).reshape(g * g, c))   # rows q1*G + q0
    st = torch.from_numpy(s).cuda()
    got = plan.fft_adjoint_image(torch.from_numpy(internal).cuda(), st).cpu().numpy()
    coils = plan.fft_adjoint_image(torch.from_numpy(internal).cuda()).cpu().numpy()
    d = okb.deapodization(n, g, j)
    shift = 0 if layout == "reference" else n // 2
    full = np.fft.ifft2(grid.astype(np.complex128)) * g * g
    pos = (np.arange(n) - shift) % g
    img = full[:, pos[:, None], pos[None, :]] * d[None]
    assert rel_l2(coils, img) <= 2e-5
    assert rel_l2(got, np.sum(np.conj(s) * img, axis=0)) <= 2e-5


# Line FFTs at every radix plan (two passes: 128, 256; three: 384, 512, 640, 1024) and coil
# grouping (16 coils: two CTAs), with image sizes beside half the grid, full grids, and image
# rows too long for the row stages' shared-memory staging.
@pytest.mark.parametrize("n,g,c", [(60, 128, 16), (128, 128, 4), (100, 256, 12), (256, 256, 8), (188, 384, 16),
                                   (260, 512, 4), (512, 512, 16), (300, 640, 8), (412, 1024, 4), (512, 1024, 12)])
def test_line_fft_endpoints_at_ragged_sizes(n, g, c):
    from trajsparsenufft_b200 import synth
    from trajsparsenufft_b200.operator import Plan
    plan = Plan.from_trajectory(synth.golden_radial(4, 32), im_size=n, grid_size=g, coils=c, width=4)
    rng = np.random.default_rng(n)
    cplx = lambda *sh: (rng.standard_normal(sh) + 1j * rng.standard_normal(sh)).astype(np.complex64)
    x, s, grid = cplx(n, n), cplx(c, n, n), cplx(c, g, g)
    d, shift = okb.deapodization(n, g, 4), n // 2
    panel, scale = plan.fft_forward_panel(torch.from_numpy(x).cuda(), torch.from_numpy(s).cuda())
    p = panel.float().cpu().numpy().astype(np.float64)
    v = (p[:, : 2 * c] + p[:, 2 * c:]).reshape(g, g, c, 2)
    got = (v[..., 0] + 1j * v[..., 1]).transpose(2, 1, 0) / scale
    assert rel_l2(got, np.fft.fft2(_grid_from_image(x[None].astype(np.complex128) * s * d[None], g, shift))) <= 1e-5
    internal = torch.from_numpy(np.ascontiguousarray(grid.transpose(2, 1, 0).reshape(g * g, c))).cuda()
    full = np.fft.ifft2(grid.astype(np.complex128)) * g * g
    pos = (np.arange(n) - shift) % g
    img = full[:, pos[:, None], pos[None, :]] * d[None]
    assert rel_l2(plan.fft_adjoint_image(internal).cpu().numpy(), img) <= 2e-5
    assert rel_l2(plan.fft_adjoint_image(internal, torch.from_numpy(s).cuda()).cpu().numpy(),
                  np.sum(np.conj(s) * img, axis=0)) <= 2e-5
