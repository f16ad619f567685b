"""FDK's ramp filter at the row lengths where its FFT changes shape: the
smallest, those around a power of two (2R-1 points at least: one more point
doubles the transform), every last radix (8, 4, 2), an odd number of rows, and
rows too long for the FFT (the Toeplitz product).  Against the oracle's FDK
(FP64 taps, direct sums) within 1e-4 of its maximum, as the FDK parity test."""
import numpy as np
import pytest

from scan_configs import ctr_desc, og_desc_xyz

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("nu", [4, 5, 16, 17, 32, 33, 64, 65, 100, 4096, 4097])
def test_fdk_row_lengths(nu, oracle_built):
    import gpu_b200
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    cfg = dict(nx=10, ny=10, nz=6, nu=nu, nv=7, nviews=3, vx=1.0, du=1.6, dso=1000.0, dod=-500.0)
    if nu > 1000:
        cfg.update(nv=5, nviews=1, nz=2)
    g = gpu_b200.Geometry(ctr_desc(cfg))
    d = og_desc_xyz(cfg)
    o = oracle_built.Oracle(d)
    b = np.random.default_rng(nu).standard_normal((cfg["nviews"],) + o.view_shape).astype(np.float32)
    vol = torch.zeros(o.vol_shape, device="cuda")
    g.fdk(torch.from_numpy(b).cuda(), vol)
    ref = o.fdk(b)
    assert np.abs(ref).max() > 0
    assert np.abs(vol.cpu().numpy() - ref).max() <= 1e-4 * np.abs(ref).max()
