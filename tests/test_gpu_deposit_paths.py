"""accumulate_rho's routes give the same bits: the one-launch deposit of small calls (up to
200,000 particles and 51,200 cells), the count and rounding kernels of larger ones, and those
of the allocation-free entry point, against np.add.at's float32 result; and the conduction
sweep's 16-byte route against its scalar one.

A cell's charge is a sequential sum of equal addends, so a deposit split into several calls
equals one call: large counts are compared with themselves in small calls."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def torch_cuda():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return torch


def _cloud(torch, n, ny, nx, dx, kind, offset, seed):
    rng = np.random.default_rng(seed)
    Lx, Ly = (nx - 1) * dx, (ny - 1) * dx
    x = rng.uniform(-0.1 * Lx, 1.1 * Lx, n)
    y = rng.uniform(-0.1 * Ly, 1.1 * Ly, n)
    if kind == "onecell":
        x[:], y[:] = 0.4 * Lx, 0.4 * Ly
    elif kind == "sorted":
        order = np.lexsort((x, np.round(y / dx)))
        x, y = x[order], y[order]
    elif kind == "halves":
        x = dx * (np.floor(x / dx) + 0.5)  # rounding ties
    x, y = x.astype(np.float32), y.astype(np.float32)
    if n > 20:
        x[3], y[5], x[7], y[9] = np.nan, np.nan, np.inf, -np.inf
    out = []
    for v in (x, y):
        t = torch.zeros(n + offset, dtype=torch.float32, device="cuda")[offset:]
        t.copy_(torch.from_numpy(v))
        out.append(t)
    return x, y, out


@pytest.mark.parametrize("kind", ["uniform", "onecell", "sorted", "halves"])
@pytest.mark.parametrize("n,ny,nx,offset", [(1, 3, 3, 0), (33, 65, 284, 0), (4097, 160, 320, 1), (199_999, 160, 320, 0),
                                            (200_000, 160, 320, 0), (200_001, 160, 320, 0), (100_003, 160, 321, 0),
                                            (300_002, 65, 284, 1), (1_000_003, 257, 1025, 0)])
def test_deposit_routes(torch_cuda, n, ny, nx, offset, kind):
    torch = torch_cuda
    import ctypes as C
    from thruster_cx_code_b200 import _lib
    from thruster_cx_code_b200.physics_engine import accumulate_rho
    dx, cd = 0.0125, 1.602e-19 * 1e17 / 80.0
    x, y, (tx, ty) = _cloud(torch, n, ny, nx, dx, kind, offset, n)
    rng = np.random.default_rng(n + 1)
    rho0 = (rng.integers(-3, 40, (ny, nx)) * np.float32(cd)).astype(np.float32)
    got = [torch.tensor(rho0, device="cuda") for _ in range(3)]
    for sign in (1.0, -1.0):
        accumulate_rho(tx, ty, got[0], n, dx, dx, nx, ny, sign * cd)
        for k in range(0, n, 65_537):
            px, py = tx[k:k + 65_537], ty[k:k + 65_537]
            accumulate_rho(px, py, got[1], px.numel(), dx, dx, nx, ny, sign * cd)
        _lib.check(_lib.load().pb_accumulate_rho_noalloc(C.c_void_p(tx.data_ptr()), C.c_void_p(ty.data_ptr()),
                                                         C.c_void_p(got[2].data_ptr()), n, dx, dx, nx, ny, sign * cd,
                                                         torch.cuda.current_stream().cuda_stream), "noalloc")
    torch.cuda.synchronize()
    ref = rho0.copy()
    with np.errstate(invalid="ignore"):
        ix = np.clip(np.round(x / np.float32(dx)).astype(np.int32), 1, nx - 2)
        iy = np.clip(np.round(y / np.float32(dx)).astype(np.int32), 1, ny - 2)
    for sign in (1.0, -1.0):
        np.add.at(ref, (iy, ix), sign * cd)
    for g in got:
        np.testing.assert_array_equal(g.cpu().numpy().view(np.uint32), ref.view(np.uint32))


@pytest.mark.parametrize("ny,nx", [(1, 1), (1, 3), (5, 7), (64, 65), (131, 257), (513, 2049)])
def test_conduction_routes(torch_cuda, ny, nx):
    torch = torch_cuda
    from thruster_cx_code_b200.physics_engine import thermal_conduction
    rng = np.random.default_rng(ny * nx)
    N = ny * nx
    T = rng.uniform(250.0, 900.0, N).astype(np.float32)
    T[::97] = np.nan
    mask = rng.integers(0, 3, N).astype(np.int32)  # values other than 0 and 1 are not the mask's
    out = []
    for off in (0, 1):
        t = torch.zeros(N + off, dtype=torch.float32, device="cuda")[off:]
        m = torch.zeros(N + off, dtype=torch.int32, device="cuda")[off:]
        d = torch.zeros(N + off, dtype=torch.float32, device="cuda")[off:]
        t.copy_(torch.from_numpy(T))
        m.copy_(torch.from_numpy(mask))
        thermal_conduction(t, d, m, nx, ny, 0.2, 0.15)
        thermal_conduction(d, t, m, nx, ny, 0.2, 0.15)
        out += [d.cpu().numpy(), t.cpu().numpy()]
    for a, b in zip(out[:2], out[2:]):
        np.testing.assert_array_equal(np.isnan(a), np.isnan(b))
        ok = ~np.isnan(a)
        np.testing.assert_array_equal(a[ok].view(np.uint32), b[ok].view(np.uint32))
