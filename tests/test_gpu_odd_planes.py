"""Volumes whose plane tables have an odd total length (nx + ny odd): the
backprojectors keep the row table (8-byte entries) beside the plane tables in
shared memory, so its place must stay 8-byte aligned for every size."""
import numpy as np
import pytest

from scan_configs import ctr_desc, og_desc_xyz

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

ODD_SUM = [dict(nx=17, ny=14, nz=11, nu=26, nv=15, nviews=6, vx=1.0, du=1.6, dso=1000.0, dod=-500.0),
           dict(nx=14, ny=17, nz=12, nu=25, nv=16, nviews=6, vx=1.0, du=1.6, dso=1000.0, dod=-500.0, initial_angle=2.0)]


@pytest.mark.parametrize("cfg", ODD_SUM, ids=["17x14x11", "14x17x12"])
def test_backprojectors_with_odd_plane_totals(cfg, oracle_built):
    import gpu_b200
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    g = gpu_b200.Geometry(ctr_desc(cfg))
    o = oracle_built.Oracle(og_desc_xyz(cfg))
    rng = np.random.default_rng(2)
    y = rng.standard_normal((cfg["nviews"],) + o.view_shape).astype(np.float32)
    vol = torch.zeros(o.vol_shape, device="cuda")
    g.backproject(torch.from_numpy(y).cuda(), vol)
    ref = o.adjoint(y)
    assert np.abs(vol.cpu().numpy() - ref).max() <= 1e-6 * np.abs(ref).max()
    # SART, bit for bit against the oracle's gather: the column walk (linear
    # and tiled volume) and the fixed-shape kernel
    truth = rng.uniform(0, 0.05, o.vol_shape).astype(np.float32)
    b = np.stack([o.forward_view(truth, j, 0) for j in range(cfg["nviews"])])
    want = np.zeros(o.vol_shape, np.float32)
    for j in range(cfg["nviews"]):
        want = o.backproject_gather(want, o.forward_view(want, j, 1, b[j]), j, 0.8)
    for bp_shape, flags in ((1, 0), (1, gpu_b200.SART_TILED), (-1, 0)):
        g.set_shapes(1, bp_shape)
        x = torch.zeros(o.vol_shape, device="cuda")
        g.sart_pass(x, torch.from_numpy(b).cuda(), 0.8, flags=flags)
        assert np.array_equal(x.cpu().numpy().view(np.uint32), np.asarray(want, np.float32).view(np.uint32)), (bp_shape, flags)
