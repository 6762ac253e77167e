"""accumulate_rho at the lines between its routes, on grids that fit a block's shared memory (at most
51,200 cells): one cluster up to 100,000 particles, the count kernels between, eighteen clusters from
1,000,000 particles on; against np.add.at's float32 result, bit for bit.  The allocation-free entry
point takes the count kernels at every size."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def torch_cuda():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return torch


@pytest.mark.parametrize("kind", ["uniform", "onecell", "sorted"])
@pytest.mark.parametrize("n,ny,nx,offset", [(99_999, 160, 320, 0), (100_000, 160, 320, 0), (100_001, 160, 320, 0),
                                            (100_000, 65, 284, 1), (100_001, 65, 284, 1),
                                            (999_999, 65, 284, 0), (1_000_000, 65, 284, 0), (1_000_003, 65, 284, 0),
                                            (1_000_001, 65, 284, 1), (1_100_001, 160, 320, 0), (1_100_001, 160, 321, 0),
                                            (1_000_000, 3, 3, 0), (2_500_000, 129, 130, 0)])
def test_lines(torch_cuda, n, ny, nx, offset, kind):
    torch = torch_cuda
    from thruster_cx_code_b200 import _lib
    from thruster_cx_code_b200.physics_engine import accumulate_rho
    rng = np.random.default_rng(n + nx)
    dx, cd = 0.0125, 1.602e-19 * 1e17 / 80.0
    x = rng.uniform(-0.1, 1.1, n) * (nx - 1) * dx
    y = rng.uniform(-0.1, 1.1, n) * (ny - 1) * dx
    if kind == "onecell":
        x[:], y[:] = x[0], y[0]
    elif kind == "sorted":
        order = np.lexsort((x, np.round(y / dx)))
        x, y = x[order], y[order]
    x, y = x.astype(np.float32), y.astype(np.float32)
    x[3], y[5], x[7], y[9] = np.nan, np.nan, np.inf, -np.inf
    dev = [torch.zeros(n + offset, dtype=torch.float32, device="cuda")[offset:] for _ in range(2)]
    for t, v in zip(dev, (x, y)):
        t.copy_(torch.from_numpy(v))
    ref = (rng.integers(-3, 40, (ny, nx)) * np.float32(cd)).astype(np.float32)
    got = [torch.tensor(ref, device="cuda") for _ in range(2)]
    for sign in (1.0, -1.0, 1.0):
        accumulate_rho(*dev, got[0], n, dx, dx, nx, ny, sign * cd)
        _lib.check(_lib.load().pb_accumulate_rho_noalloc(
            *[C.c_void_p(t.data_ptr()) for t in (*dev, got[1])], n, dx, dx, nx, ny, sign * cd,
            torch.cuda.current_stream().cuda_stream), "noalloc")
    torch.cuda.synchronize()
    with np.errstate(invalid="ignore"):
        ix = np.clip(np.round(x / np.float32(dx)).astype(np.int32), 1, nx - 2)
        iy = np.clip(np.round(y / np.float32(dx)).astype(np.int32), 1, ny - 2)
    for sign in (1.0, -1.0, 1.0):
        np.add.at(ref, (iy, ix), sign * cd)
    for g in got:
        np.testing.assert_array_equal(g.cpu().numpy().view(np.uint32), ref.view(np.uint32))
