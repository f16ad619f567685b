"""FDK's ramp filter at the row lengths where its FFT changes shape: the
smallest, those around a power of two (2R-1 points at least: one more point
doubles the transform), every last radix (8, 4, 2), an odd number of rows, and
rows too long for the FFT (the Toeplitz product).  The voxels read the rows
from end to end, where a transform one point short would show.  Against the
oracle's FDK (FP64 taps, direct sums rounded to FP32)."""
import numpy as np
import pytest

from scan_configs import ctr_desc, og_desc_xyz

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("nu", [4, 5, 8, 9, 16, 17, 32, 33, 64, 65, 100, 500, 1024, 1025, 4096, 4097])
def test_fdk_row_lengths(nu, oracle_built):
    """One slice as wide as the detector sees, so that every column is read.  Random rows: the filter's FP32 rounding and
    the backprojection's, 2e-6 of the largest voxel (1e-5 for the Toeplitz product's 4097 FP32 terms).  Impulses at both
    ends of a row, one view: the far columns hold the taps of the longest lags, 1e-3 to 1e-7 of the largest, each to
    some ten FP32 roundings of itself."""
    import gpu_b200
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    n = max(10, min(nu, 200))
    cfg = dict(nx=n, ny=n, nz=1, nu=nu, nv=7, nviews=3, vx=200.0 / n, du=1.5 * 200.0 / nu, dso=1000.0, dod=-500.0)

    def both(cfg, b):
        o = oracle_built.Oracle(og_desc_xyz(cfg))
        vol = torch.zeros(o.vol_shape, device="cuda")
        gpu_b200.Geometry(ctr_desc(cfg)).fdk(torch.from_numpy(b).cuda(), vol)
        return vol.cpu().numpy(), o.fdk(b)

    got, ref = both(cfg, np.random.default_rng(nu).standard_normal((3, 7, nu)).astype(np.float32))
    top = np.abs(ref).max()
    assert top > 0 and np.abs(got - ref).max() <= (2e-6 if nu <= 4096 else 1e-5) * top
    for at in (0, nu - 1):
        b = np.zeros((1, 7, nu), np.float32)
        b[:, :, at] = 1.0
        got, ref = both(dict(cfg, nviews=1), b)
        err, mag = np.abs(got - ref), np.abs(ref)
        far = mag <= 1e-3 * mag.max()
        assert mag.max() > 0 and np.all(err <= 1e-6 * mag.max())
        assert np.all(err[far] <= 1e-6 * mag[far] + 1e-12 * mag.max())


def rows_scan(nu, nv):
    """A thin column of voxels whose slices read every detector row, four slices a row."""
    cfg = dict(nx=4, ny=4, nz=4 * nv, nu=nu, nv=nv, nviews=3, vx=0.25, du=1.5, dso=1000.0, dod=-500.0)
    return cfg, og_desc_xyz(cfg)


def both(cfg, o, b):
    import gpu_b200
    vol = torch.zeros(o.vol_shape, device="cuda")
    gpu_b200.Geometry(ctr_desc(cfg)).fdk(torch.from_numpy(b).cuda(), vol)
    return vol.cpu().numpy(), o.fdk(b)


@pytest.mark.parametrize("nu,nv", [(16, 8), (100, 7), (1000, 8), (4097, 5)])
def test_fdk_rows_are_filtered_alone(nu, nv, oracle_built):
    """A detector row's values reach the voxels that read that row and no others: a NaN, an Inf, rows 1e4 times their
    neighbours, rows of zeros, for an even and an odd number of rows.  The oracle's filter is a direct FP64 sum per
    row.  Rows of a transform (nu <= 4096) come out correctly rounded but for rare ties, so voxels agree to the
    backprojection's own rounding: 1e-6 of the largest among them."""
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    cfg, d = rows_scan(nu, nv)
    o = oracle_built.Oracle(d)
    rng = np.random.default_rng(nu)
    b = rng.standard_normal((3,) + o.view_shape).astype(np.float32)
    clean, ref = both(cfg, o, b)
    tol = 1e-6 if nu <= 4096 else 1e-5   # a Toeplitz product of 4097 FP32 terms
    assert np.abs(clean - ref).max() <= tol * np.abs(ref).max()
    for bad in (np.nan, np.inf, -np.inf):
        for w, v in ((1, 2), (2, nv - 1), (0, 0)):
            c = b.copy()
            c[w, v, nu // 3] = bad
            got, want = both(cfg, o, c)
            hit = ~np.isfinite(want)
            assert hit.any() and not hit.all()
            assert np.array_equal(~np.isfinite(got), hit), (bad, w, v)
            assert np.array_equal(got[~hit], clean[~hit]), (bad, w, v)
    strong = np.zeros(b.shape, bool)
    strong[:, np.arange(nv) % 4 % 3 == 0] = True    # rows s w w s s w w s ...
    only = both(cfg, o, np.where(strong, b, np.float32(0)))
    quiet = only[1] == 0.0                           # voxels between two weak rows
    assert quiet.any() and not quiet.all()
    assert not only[0][quiet].any()
    got, want = both(cfg, o, np.where(strong, np.float32(1e4), np.float32(1)) * b)
    assert np.abs(got - want)[quiet].max() <= tol * np.abs(want[quiet]).max()


def test_fdk_smooth_rows(oracle_built):
    """Rows that are nearly constant: what the ramp leaves is small against the row, and is still right to FP32."""
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    cfg, d = rows_scan(1024, 6)
    o = oracle_built.Oracle(d)
    u = np.linspace(-1, 1, 1024)
    b = (5.0 + np.exp(-u ** 2) + 0.01 * np.cos(40 * u))[None, None, :] * (1.0 + 0.1 * np.arange(6))[None, :, None]
    got, want = both(cfg, o, np.repeat(b, 3, 0).astype(np.float32))
    assert np.abs(got - want).max() <= 1e-6 * np.abs(want).max()


@pytest.mark.parametrize("us", [360.0 / 3, 0.5])
@pytest.mark.parametrize("shape", [(57, 148, 64), (61, 150, 40), (57, 144, 64), (7, 3, 33), (3, 5, 33), (1, 1, 1)])
def test_fdk_backprojection_shapes(shape, us, oracle_built):
    """The backprojection with 8 and with 4 voxels a thread (592 blocks of 8 and just below, few slices), a full circle
    and a short scan, bit for bit against the reference kernel's arithmetic."""
    import gpu_b200
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    nz, ny, nx = shape
    cfg = dict(nx=nx, ny=ny, nz=nz, nu=90, nv=40, nviews=3, vx=1.0, du=2.0, dso=1000.0, dod=-500.0, initial_angle=2.0)
    d = ctr_desc(cfg)
    d.us_rate = us
    od = og_desc_xyz(cfg)
    od.us_rate = us
    o = oracle_built.Oracle(od)
    rng = np.random.default_rng(5)
    filt = rng.standard_normal((3,) + o.view_shape).astype(np.float32)
    want = rng.uniform(0, 1, o.vol_shape).astype(np.float32)
    vol = torch.from_numpy(want.copy()).cuda()
    gpu_b200.Geometry(d).fdk_backproject(torch.from_numpy(filt).cuda(), vol)
    for j in range(3):
        want = o.fdk_bp_view(want, filt[j], j)
    assert np.array_equal(vol.cpu().numpy().view(np.uint32), np.asarray(want, np.float32).view(np.uint32))
