"""The FGP-TV prox at the edges of its blocks: volumes one voxel short of, at
and past a 32 x 8 tile and a run of z planes, single planes, rows and voxels,
runs of 4 to 32 planes.  Bit for bit against the same float operations in
numpy, the duals rounded to the storage type (FP32 and FP16) after each step
(V63/kernel_FGP_Denoise_GPUx7.cu:2-88)."""
import numpy as np
import pytest

from kernels_run import kernels_run, none_of

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
F = np.float32


def prox(f, lam, iters, dt):
    lam = F(lam)
    f = f.astype(dt).astype(F)
    axes = (2, 1, 0)   # r along x, s along y, t along z
    cur = [np.zeros(f.shape, F) for _ in axes]
    old = [np.zeros(f.shape, F) for _ in axes]

    def back(a, ax):   # the dual of the previous edge, 0 before the first
        out = np.zeros_like(a)
        hi = [slice(None)] * 3
        lo = [slice(None)] * 3
        hi[ax], lo[ax] = slice(1, None), slice(None, -1)
        out[tuple(hi)] = a[tuple(lo)]
        return out

    def L(d):
        r, s, t = (d[i] - back(d[i], ax) for i, ax in enumerate(axes))
        return f - lam * ((r + s) + t)

    a12 = F(1.0) / (lam * F(12.0))
    t0 = F(1.0)
    for _ in range(iters):
        t1 = (F(1.0) + np.sqrt(F(1.0) + F(4.0) * t0 * t0)) / F(2.0)
        gam = (t0 - F(1.0)) / t1
        l = L(cur)
        v = []
        for i, ax in enumerate(axes):
            nxt = np.zeros_like(l)
            n = l.shape[ax]
            sl = [slice(None)] * 3
            up = [slice(None)] * 3
            sl[ax], up[ax] = slice(0, n - 1), slice(1, n)
            step = np.zeros_like(l)
            step[tuple(sl)] = a12 * (l[tuple(sl)] - l[tuple(up)])
            inner = np.zeros(l.shape, bool)
            inner[tuple(sl)] = True
            v.append((np.where(inner, cur[i] + step, cur[i]), inner))
        den = np.maximum(F(1.0), np.sqrt((v[0][0] * v[0][0] + v[1][0] * v[1][0]) + v[2][0] * v[2][0]))
        for i in range(3):
            on = v[i][0] / den
            inner = v[i][1]
            cur[i] = np.where(inner, (on + gam * (on - old[i])).astype(dt).astype(F), F(0.0))
            old[i] = np.where(inner, on.astype(dt).astype(F), F(0.0))
        t0 = t1
    return L(old).astype(dt)


@pytest.mark.parametrize("dtype", ["f32", "f16"])
@pytest.mark.parametrize("shape", [(1, 1, 1), (1, 1, 40), (3, 1, 1), (4, 8, 32), (5, 9, 33), (3, 7, 31), (33, 16, 64),
                                   (70, 17, 65), (2, 300, 5)])
def test_fgp_block_edges(shape, dtype):
    import gpu_b200
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    nz, ny, nx = shape
    dt = {"f32": np.float32, "f16": np.float16}[dtype]
    g = gpu_b200.Geometry(gpu_b200.make_desc(nx, ny, nz, 0.5, 16, 16, 1.0, 1000.0, -1000.0, 4))
    rng = np.random.default_rng(nx + 100 * ny)
    vol = (rng.uniform(0, 0.05, shape) + 0.2 * (rng.random(shape) > 0.9)).astype(dt)
    for lam, iters in ((0.01, 1), (0.01, 2), (0.01, 7), (1e-4, 3)):
        x = torch.from_numpy(vol.copy()).cuda()
        g.fgp_tv(x, lam, iters)
        want = prox(vol, lam, iters, dt)
        got = x.cpu().numpy()
        assert np.array_equal(got, want), (lam, iters, np.abs(got.astype(F) - want.astype(F)).max())


def run(shape, dtype, lam_iters, form):
    import gpu_b200
    nz, ny, nx = shape
    dt = {"f32": np.float32, "f16": np.float16}[dtype]
    g = gpu_b200.Geometry(gpu_b200.make_desc(nx, ny, nz, 0.1, 16, 16, 1.0, 1000.0, -1000.0, 4))
    rng = np.random.default_rng(nx + 100 * ny)
    vol = (rng.uniform(0, 0.05, shape) + 0.2 * (rng.random(shape) > 0.9)).astype(dt)
    names = kernels_run(lambda: g.fgp_tv(torch.from_numpy(vol.copy()).cuda(), 0.01, 2))
    assert none_of(names, *(("k_fgp_L", "k_fgp_dual") if form == "one pass" else ("k_fgp_step",))), names
    for lam, iters in lam_iters:
        x = torch.from_numpy(vol.copy()).cuda()
        g.fgp_tv(x, lam, iters)
        want = prox(vol, lam, iters, dt)
        assert np.array_equal(x.cpu().numpy(), want), (lam, iters)


@pytest.mark.parametrize("dtype", ["f32", "f16"])
@pytest.mark.parametrize("shape,form", [
    # one pass: full tiles, a voxel short of and past them, runs of 4 planes and remainders
    ((4, 8, 32), "one pass"), ((9, 16, 65), "one pass"), ((35, 15, 63), "one pass"), ((5, 25, 64), "one pass"),
    ((33, 33, 97), "one pass"), ((2, 40, 96), "one pass"), ((1, 7, 31), "one pass"), ((6, 9, 33), "one pass"),
    # two: tiles mostly empty
    ((33, 33, 33), "two passes"), ((40, 1, 900), "two passes"), ((90, 80, 5), "two passes"), ((40, 9, 129), "two passes")])
def test_fgp_forms(shape, form, dtype):
    """The one-pass and the two-pass iteration, each where the rule takes it."""
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    run(shape, dtype, ((0.01, 1), (0.01, 2), (0.01, 5), (1e-4, 3)), form)


@pytest.mark.parametrize("shape,dtype,form", [((1, 1024, 1024), "f32", "two passes"), ((2, 1024, 1024), "f16", "two passes"),
                                              ((2, 1300, 1300), "f32", "one pass"), ((400, 504, 16), "f32", "one pass"),
                                              ((400, 504, 16), "f16", "two passes")])
def test_fgp_forms_large(shape, dtype, form):
    """Few planes and half-filled tiles, on both sides of the size at which the duals exceed the L2 cache."""
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    run(shape, dtype, ((0.01, 2),), form)


def test_fgp_in_short_memory():
    """Where nine dual arrays do not fit the memory the prox runs in two passes on six and L: the same bits."""
    import gpu_b200
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    n = (256, 512, 512)
    desc = gpu_b200.make_desc(n[2], n[1], n[0], 0.1, 16, 16, 1.0, 1000.0, -1000.0, 4)
    vol = torch.rand(n, device="cuda", generator=torch.Generator(device="cuda").manual_seed(2))
    g = gpu_b200.Geometry(desc)
    want = g.fgp_tv(vol.clone(), 0.01, 3)
    g.close()
    got = vol.clone()
    g = gpu_b200.Geometry(desc)
    # the two-pass kernels are loaded before the memory is taken
    gpu_b200.Geometry(gpu_b200.make_desc(1024, 1024, 1, 0.1, 16, 16, 1.0, 1000.0, -1000.0, 4)).fgp_tv(
        torch.rand((1, 1024, 1024), device="cuda"), 0.01, 1)
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    V = vol.numel()
    hold = torch.empty(torch.cuda.mem_get_info()[0] - 32 * V, dtype=torch.uint8, device="cuda")   # between 28 V and 36 V left
    try:
        g.fgp_tv(got, 0.01, 3)
        assert torch.equal(got, want)
        names = kernels_run(lambda: g.fgp_tv(got, 0.01, 1))
        assert none_of(names, "k_fgp_step"), names
    finally:
        del hold
        torch.cuda.empty_cache()
