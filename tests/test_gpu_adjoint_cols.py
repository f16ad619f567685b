"""The matched adjoint at the edges of the z-column gather's tiles and rule: volumes one voxel short of,
at and past 8 x 4 columns and 32 slices, a single voxel, detector columns much
finer than a voxel (runs longer than the four a column keeps) and coarser,
steep cones, accumulation, 16-bit volumes.  Against the oracle's scatter of the
projector's own segments in FP64, to float rounding (as the parity test)."""
import numpy as np
import pytest

from kernels_run import kernels_run, none_of
from scan_configs import ctr_desc, og_desc_xyz

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def scan(nx, ny, nz, **kw):
    return dict(dict(nx=nx, ny=ny, nz=nz, nu=29, nv=23, nviews=9, vx=1.0, du=1.3, dso=1000.0, dod=-500.0), **kw)


SCANS = {
    "8x4x32": scan(8, 4, 32), "9x5x33": scan(9, 5, 33, initial_angle=1.0), "7x3x31": scan(7, 3, 31),
    "one": scan(1, 1, 1, du=0.2), "17x6x65": scan(17, 6, 65, nv=60), "slice": scan(24, 20, 1, nv=5),
    "fine": scan(9, 8, 6, nu=130, nv=70, du=0.19), "coarse": scan(30, 29, 20, nu=9, nv=7, du=7.0),
    # an odd number of rays in a batch, axis-parallel and on-plane rays among them
    "odd_rays": scan(12, 12, 12, nu=17, nv=13, nviews=7, du=1.6),
    "odd_planes": scan(11, 12, 11, nu=17, nv=13, nviews=1, du=1.5),
    # the slices at which the gather starts (7 / 8, fan and parallel beams 11 / 12), and warps of a block: 1, 2, 3 x 2
    "7_slices": scan(34, 20, 7), "8_slices": scan(34, 20, 8), "11_fan": scan(33, 18, 11, ct_style=1),
    "12_fan": scan(33, 18, 12, ct_style=1), "12_parallel": scan(33, 18, 12, ct_style=2), "40_slices": scan(9, 9, 40, nv=60),
    "129_slices": scan(9, 5, 129, nv=90, du=2.0),
    "steep": scan(12, 10, 70, nu=24, nv=90, du=1.4, dso=30.0, dod=-30.0, initial_angle=3.0),
}


@pytest.mark.parametrize("name", sorted(SCANS))
def test_adjoint_tile_edges(name, oracle_built):
    import gpu_b200
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    cfg = SCANS[name]
    g = gpu_b200.Geometry(ctr_desc(cfg))
    o = oracle_built.Oracle(og_desc_xyz(cfg))
    y = np.random.default_rng(3).standard_normal((cfg["nviews"],) + o.view_shape).astype(np.float32)
    ref = o.adjoint(y)
    dy = torch.from_numpy(y).cuda()
    vol = torch.full(o.vol_shape, 7.0, device="cuda")
    names = kernels_run(lambda: g.backproject(dy, vol))        # overwrites
    gather = cfg["nz"] >= (12 if cfg.get("ct_style") else 8)
    assert none_of(names, *(("k_adjoint", "k_ray_prep") if gather else ("k_adj_cols", "k_adj_prep"))), names
    got = vol.cpu().numpy().astype(np.float64)
    top = np.abs(ref).max()
    assert top > 0
    assert np.all(np.abs(got - ref) <= 1.2e-7 * np.abs(ref) + 1e-12 * top)
    g.backproject(dy, vol, flags=gpu_b200.BP_ACCUMULATE)       # one rounding of the sum
    assert np.all(np.abs(vol.cpu().numpy() - 2.0 * got) <= 2.4e-7 * np.abs(ref) + 1e-12 * top)
    half = torch.zeros(o.vol_shape, device="cuda", dtype=torch.bfloat16)
    g.backproject(dy, half)
    assert torch.equal(half.cpu(), torch.from_numpy(got.astype(np.float32)).to(torch.bfloat16))


def test_adjoint_workspace_does_not_depend_on_the_call(oracle_built):
    """The first call reserves a whole batch's ray records (about 256 MB at most), so a longer call neither allocates
    nor moves them, and a captured short call can be replayed after it."""
    import gpu_b200
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    cfg = scan(40, 36, 33, nu=512, nv=400, nviews=45, du=0.2)
    g = gpu_b200.Geometry(ctr_desc(cfg))
    gen = torch.Generator(device="cuda").manual_seed(1)
    y = torch.randn((45,) + g.view_shape, device="cuda", generator=gen)
    long = torch.empty(g.vol_shape, device="cuda")
    one = torch.empty(g.vol_shape, device="cuda")
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    g.backproject(y[7:8], one, 7, 1)
    torch.cuda.synchronize()
    first = torch.cuda.mem_get_info()[0]
    assert before - first <= (256 << 20) + 512 * 64 * 8 + (4 << 20)   # records, marks, granularity
    graph = torch.cuda.CUDAGraph()
    out = torch.zeros_like(one)
    with torch.cuda.graph(graph):
        g.backproject(y[7:8], out, 7, 1)
    torch.cuda.synchronize()
    first = torch.cuda.mem_get_info()[0]
    g.backproject(y, long)
    torch.cuda.synchronize()
    assert torch.cuda.mem_get_info()[0] == first   # (checked before the replay: it would use freed memory)
    out.zero_()
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(out, one)


@pytest.mark.parametrize("n", [96, 112])
def test_adjoint_irregular_rays(n, oracle_built):
    """An axis-aligned view where rays enter the volume within rounding of voxel edges (263 of 20,736 rays at 96^3, one
    to three in most detector columns; 20 at 112^3), on more than 64 rows.  The traversal of such a ray may begin with a
    segment as long as the rounding of its entry alpha, 2^-23 of the ray's length, which the gather leaves with the next
    voxel: that, times the value, is the tolerance beside the regular rays' (test_adjoint_tile_edges)."""
    import gpu_b200
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    p = 256.0 / n
    cfg = scan(n, n, n, nu=n * 3 // 2, nv=n * 3 // 2, nviews=1, vx=p, du=p)
    g = gpu_b200.Geometry(ctr_desc(cfg))
    o = oracle_built.Oracle(og_desc_xyz(cfg))
    y = np.random.default_rng(3).standard_normal((1,) + o.view_shape).astype(np.float32)
    ref = o.adjoint(y)
    vol = torch.zeros(o.vol_shape, device="cuda")
    g.backproject(torch.from_numpy(y).cuda(), vol)
    d12 = float(np.hypot(1500.0, 0.5 * cfg["nu"] * p * 2 ** 0.5))
    err = np.abs(vol.cpu().numpy() - ref)
    assert np.all(err <= 1.2e-7 * np.abs(ref) + 2.0 ** -23 * d12 * np.abs(y).max())
    assert (err > 1.2e-7 * np.abs(ref) + 1e-12 * np.abs(ref).max()).sum() <= 1e-3 * ref.size
