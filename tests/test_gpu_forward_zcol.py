"""ctr_forward on a z-column copy of the volume (calls of many rays) against the
general projector (the same views one at a time, below that size), bit for bit:
every scanner, odd and even detectors, exact 0/45/90-degree views (rays on
planes, x and y planes crossed at one alpha), wide cones (rays entering and
leaving through the z faces, several z planes a step), lists long enough for
two columns a block, a volume touching the detector plane, offsets, the three storage types, fused sums, NaN voxels, and
1 to 33 slices."""
import numpy as np
import pytest

from scan_configs import NEAR_DETECTOR, SLABS, SMALL, STYLES, TBCT, ctr_desc, view_rows

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

LIST = dict(SMALL, near_detector=NEAR_DETECTOR, cone_wide=SLABS["cone_wide"], **STYLES, **TBCT,
            square=dict(nx=20, ny=20, nz=9, nu=21, nv=7, nviews=8, vx=1.0, du=1.5, dso=1000.0, dod=-500.0, ct_style=2),
            flat=dict(nx=33, ny=17, nz=1, nu=40, nv=3, nviews=8, vx=1.0, du=1.2, dso=1000.0, dod=-500.0),
            tall=dict(nx=9, ny=40, nz=33, nu=41, nv=64, nviews=8, vx=1.0, du=1.0, dso=60.0, dod=-60.0),
            long=dict(nx=850, ny=801, nz=24, nu=60, nv=24, nviews=8, vx=0.3, du=6.0, dso=1000.0, dod=-500.0),
            steep=dict(nx=8, ny=8, nz=64, nu=16, nv=70, nviews=8, vx=1.0, du=3.0, dso=30.0, dod=-30.0))


# the path wants 480 x and y planes (900 for 16-bit voxels with the reference's
# sums), 4.5e9 rays x planes and 120 a voxel, and detector rows that fill its
# blocks: the scans' volumes are widened by more voxels of a finer pitch, the
# detector gets 127 or 128 rows over a little more than the volume's height
# (the tetrahedron beam: sources for about 60 rows), and the views repeat over
# many turns
def widened(cfg):
    f = -(-900 // (cfg["nx"] + cfg["ny"]))
    nz = cfg["nz"] * f if "n_sources" in cfg else min(cfg["nz"] * f, 40)   # (the sources' places follow the height)
    out = dict(cfg, nx=cfg["nx"] * f, ny=cfg["ny"] * f, nz=nz, vx=cfg["vx"] / f, m_offset=cfg.get("m_offset", 0) * f)
    if "n_sources" in cfg:
        out["n_sources"] = {4: 16, 3: 21, 5: 11}[cfg["nv"]]
    else:
        cone = cfg.get("ct_style", 0) == 0
        height = nz * (out["vx"] if cone else cfg["du"])
        n = 128 - cfg["nv"] % 2
        out.update(nv=n, dv=1.2 * height * ((cfg["dso"] - cfg["dod"]) / cfg["dso"] if cone else 1.0) / n)
    return out


def geometry(cfg, fast=False):
    import gpu_b200
    d = ctr_desc(cfg, fast_sums=fast)
    d.dv = cfg.get("dv", 0.0)
    return gpu_b200.Geometry(d)


def zcol_ran(make, vol, out):
    """Whether views [0, len(out)) of a new geometry took the z-column path: its scratch, a copy of the volume, stays
    with the geometry and is missing from the device's free memory.  (The first call loads the kernels.)"""
    first, new = make(), make()
    first.forward(vol, out, 0, len(out))
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    new.forward(vol, out, 0, len(out))
    torch.cuda.synchronize()
    taken = before - torch.cuda.mem_get_info()[0]
    assert taken == 0 or taken >= vol.numel() * vol.element_size(), taken
    return taken > 0


@pytest.mark.parametrize("fast", [False, True])
@pytest.mark.parametrize("name", sorted(LIST))
def test_zcol_equals_the_general_projector(name, fast):
    import gpu_b200
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    cfg = widened(LIST[name])
    rays = max(4.5e9, 120.0 * cfg["nx"] * cfg["ny"] * cfg["nz"]) / (cfg["nx"] + cfg["ny"])
    cfg["nviews"] = n = int(rays // (cfg["nu"] * view_rows(cfg)) // 8 + 1) * 8
    g = geometry(cfg, fast)
    gen = torch.Generator(device="cuda").manual_seed(4)
    base = torch.rand(g.vol_shape, device="cuda", generator=gen)
    base.view(-1)[base.numel() // 3] = float("nan")
    for dt in (torch.float32, torch.float16, torch.bfloat16):
        vol = base.to(dt)
        out = torch.zeros((n,) + g.view_shape, device="cuda")
        g.forward(vol, out)
        assert zcol_ran(lambda: geometry(cfg, fast), vol, out)
        assert not zcol_ran(lambda: geometry(cfg, fast), vol, out[:1])
        g.forward(vol, out)
        if dt != torch.float32:   # stored in 16 bits: the same sums rounded once
            half = g.forward(vol, torch.zeros(out.shape, device="cuda", dtype=dt))
            assert bool(((half == out.to(dt)) | (torch.isnan(half) & torch.isnan(out))).all())
            del half
        one = torch.zeros((1,) + g.view_shape, device="cuda")
        for j in sorted({0, 1, n // 8, n // 4, n // 4 + 1, n // 2, 5 * n // 8, n - 1}):
            g.forward(vol, one, j, 1)
            a, b = out[j].view(torch.int32), one[0].view(torch.int32)
            same = (a == b) | (torch.isnan(out[j]) & torch.isnan(one[0]))
            assert bool(same.all()), (j, dt, int((~same).sum()), float((out[j] - one[0]).abs().nan_to_num().max()))


@pytest.mark.parametrize("fast", [False, True])
def test_zcol_z_steps_as_short_as_in_plane_steps(fast):
    """A cone so wide that a ray crosses about as many z planes as x or y planes, a thousand times magnified so that the
    rounding of an alpha is a hundredth of a step: an entry of the list must not hold two z crossings."""
    import gpu_b200
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    n, nz, nu = 240, 512, 128
    views = int(4.6e9 // (2 * n * nu * nu)) + 1
    mag = 1003.5 / 3.5
    desc = gpu_b200.make_desc(n, n, nz, 0.01, nu, nu, 1.2 * n * 0.01 * mag / nu, 3.5, -1000.0, views,
                              dv=1.2 * nz * 0.01 * mag / nu, fast_sums=fast)
    g = gpu_b200.Geometry(desc)
    vol = torch.rand(g.vol_shape, device="cuda", generator=torch.Generator(device="cuda").manual_seed(3))
    out = torch.zeros((views,) + g.view_shape, device="cuda")
    one = torch.zeros((1,) + g.view_shape, device="cuda")
    assert zcol_ran(lambda: gpu_b200.Geometry(desc), vol, out)
    g.forward(vol, out)
    for j in range(0, views, 2):
        g.forward(vol, one, j, 1)
        assert torch.equal(out[j], one[0]), (j, int((out[j] != one[0]).sum()))


def test_zcol_rule():
    """Detector rows are the path's lanes, so rows that do not fill them, or do not meet the volume, keep the general
    projector: (nx = ny, nz, nu, nv, taken)."""
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    for n, nz, nu, nv, taken in ((512, 64, 1024, 64, True), (512, 32, 1024, 32, True), (512, 16, 1024, 16, False),
                                 (512, 1, 2048, 1, False), (512, 4, 1024, 64, False), (512, 64, 1024, 72, False),
                                 (512, 96, 1024, 96, True), (1024, 32, 512, 32, False), (1600, 64, 512, 256, False)):
        views = int(max(4.6e9, 121.0 * n * n * nz) / (nu * nv * 2 * n)) + 1
        cfg = dict(nx=n, ny=n, nz=nz, vx=256.0 / n, nu=nu, nv=nv, du=384.0 / nu, nviews=views, dso=1000.0, dod=-500.0,
                   dv=384.0 / n)
        g = geometry(cfg)
        vol = torch.rand(g.vol_shape, device="cuda")
        out = torch.empty((views,) + g.view_shape, device="cuda")
        assert zcol_ran(lambda: geometry(cfg), vol, out) == taken, (n, nz, nu, nv)


def test_zcol_forward_under_capture_and_on_streams():
    """A captured call takes the path without scratch; calls on two streams have their own scratch."""
    import gpu_b200
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    n = 1640
    cfg = dict(widened(SMALL["cube16"]), nviews=n)
    g = geometry(cfg)
    vols = [torch.rand(g.vol_shape, device="cuda") for _ in range(2)]
    want = [g.forward(v, torch.zeros((n,) + g.view_shape, device="cuda")) for v in vols]
    assert zcol_ran(lambda: geometry(cfg), vols[0], torch.zeros_like(want[0]))
    torch.cuda.synchronize()
    outs = [torch.zeros_like(w) for w in want]
    streams = [torch.cuda.Stream() for _ in range(2)]
    for _ in range(4):
        for v, o, s in zip(vols, outs, streams):
            g.forward(v, o, stream=s)
    torch.cuda.synchronize()
    assert all(torch.equal(a, b) for a, b in zip(outs, want))
    cap = torch.zeros_like(want[0])
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        g.forward(vols[0], cap)
    cap.zero_()
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(cap, want[0])


def test_zcol_forward_beside_another_threads_capture():
    """A call's scratch does not disturb a capture that another thread has open (in the global mode), neither the first
    call of a geometry, which makes the pool, nor a later one."""
    import threading

    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    n = 1640
    cfg = dict(widened(SMALL["cube16"]), nviews=n)
    warm, new = (geometry(cfg) for _ in range(2))
    vol = torch.rand(warm.vol_shape, device="cuda")
    side = torch.cuda.Stream()
    outs = [torch.zeros((n,) + warm.view_shape, device="cuda") for _ in range(3)]
    warm.forward(vol, outs[0])
    torch.cuda.synchronize()
    for g, out in ((warm, outs[1]), (new, outs[2])):
        failed = []

        def other():
            try:
                g.forward(vol, out, stream=side)
            except Exception as e:
                failed.append(e)

        x = torch.zeros(64, device="cuda")
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, capture_error_mode="global"):
            x += 1
            t = threading.Thread(target=other)
            t.start()
            t.join()
            x += 1
        assert not failed
        graph.replay()
        torch.cuda.synchronize()
        assert float(x.sum()) == 128.0
        assert torch.equal(out, outs[0])
