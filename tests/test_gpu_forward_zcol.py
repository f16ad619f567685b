"""ctr_forward on a z-column copy of the volume (calls of many rays) against the
general projector (the same views one at a time, below that size), bit for bit:
every scanner, odd and even detectors, exact 0/45/90-degree views (rays on
planes, x and y planes crossed at one alpha), wide cones (rays entering and
leaving through the z faces, several z planes a step), a volume touching the
detector plane, offsets, the three storage types, fused sums, NaN voxels, and
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
            steep=dict(nx=8, ny=8, nz=64, nu=16, nv=70, nviews=8, vx=1.0, du=3.0, dso=30.0, dod=-30.0))


# the path wants 480 x and y planes (900 for 16-bit voxels with the reference's
# sums), 4.5e9 rays x planes and 120 a voxel: the scans' volumes are widened by more voxels of
# a finer pitch, and the views repeat over many turns
def widened(cfg):
    f = -(-900 // (cfg["nx"] + cfg["ny"]))
    nz = cfg["nz"] * f if "n_sources" in cfg else min(cfg["nz"] * f, 40)   # (the sources' places follow the height)
    return dict(cfg, nx=cfg["nx"] * f, ny=cfg["ny"] * f, nz=nz, vx=cfg["vx"] / f, m_offset=cfg.get("m_offset", 0) * f)


@pytest.mark.parametrize("fast", [False, True])
@pytest.mark.parametrize("name", sorted(LIST))
def test_zcol_equals_the_general_projector(name, fast):
    import gpu_b200
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    cfg = widened(LIST[name])
    rays = max(4.5e9, 120.0 * cfg["nx"] * cfg["ny"] * cfg["nz"]) / (cfg["nx"] + cfg["ny"])
    cfg["nviews"] = n = int(rays // (cfg["nu"] * view_rows(cfg)) // 8 + 1) * 8
    g = gpu_b200.Geometry(ctr_desc(cfg, fast_sums=fast))
    gen = torch.Generator(device="cuda").manual_seed(4)
    base = torch.rand(g.vol_shape, device="cuda", generator=gen)
    base.view(-1)[base.numel() // 3] = float("nan")
    for dt in (torch.float32, torch.float16, torch.bfloat16):
        vol = base.to(dt)
        out = torch.zeros((n,) + g.view_shape, device="cuda")
        g.forward(vol, out)
        one = torch.zeros((1,) + g.view_shape, device="cuda")
        for j in sorted({0, 1, n // 8, n // 4, n // 4 + 1, n // 2, 5 * n // 8, n - 1}):
            g.forward(vol, one, j, 1)
            a, b = out[j].view(torch.int32), one[0].view(torch.int32)
            same = (a == b) | (torch.isnan(out[j]) & torch.isnan(one[0]))
            assert bool(same.all()), (j, dt, int((~same).sum()), float((out[j] - one[0]).abs().nan_to_num().max()))


def test_zcol_forward_under_capture_and_on_streams():
    """A captured call takes the path without scratch; calls on two streams have their own scratch."""
    import gpu_b200
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    n = 10400
    cfg = dict(widened(SMALL["cube16"]), nviews=n)
    g = gpu_b200.Geometry(ctr_desc(cfg))
    vols = [torch.rand(g.vol_shape, device="cuda") for _ in range(2)]
    want = [g.forward(v, torch.zeros((n,) + g.view_shape, device="cuda")) for v in vols]
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

    import gpu_b200
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    n = 10400
    cfg = dict(widened(SMALL["cube16"]), nviews=n)
    vol = torch.rand(gpu_b200.Geometry(ctr_desc(cfg)).vol_shape, device="cuda")
    warm, new = (gpu_b200.Geometry(ctr_desc(cfg)) for _ in range(2))
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
