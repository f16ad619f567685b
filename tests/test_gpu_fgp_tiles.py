"""The FGP-TV prox at the edges of its blocks: volumes one voxel short of, at
and past a 32 x 8 tile and a run of z planes, single planes, rows and voxels,
runs of 4 to 32 planes.  Bit for bit against the same float operations in
numpy, the duals rounded to the storage type (FP32 and FP16) after each step
(V63/kernel_FGP_Denoise_GPUx7.cu:2-88)."""
import numpy as np
import pytest

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
