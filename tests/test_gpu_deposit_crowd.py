"""accumulate_rho of particles that crowd into few cells without being sorted, where warps add equal cells
together, of particles that change from scattered to crowded or sorted along the array, and at counts
that leave lanes and turns of a warp empty; against np.add.at's float32 result, bit for bit."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _cells(rng, n, ny, nx, cells):
    """n random cells out of `cells` interior ones in a corner of the grid (0: all of them)"""
    total = (ny - 2) * (nx - 2)
    pick = rng.choice(total, size=min(cells, total), replace=False) if cells else np.arange(total)
    k = pick[rng.integers(0, len(pick), n)]
    return 1 + k // (nx - 2), 1 + k % (nx - 2)


@pytest.mark.parametrize("cells", [2, 20, 60, 250, 1000, "mixed"])
@pytest.mark.parametrize("n,ny,nx,offset", [(31, 257, 1025, 0), (1029, 257, 1025, 0), (100_003, 257, 1025, 1),
                                            (400_001, 65, 284, 0), (1_300_007, 257, 1025, 0), (2_600_002, 257, 1025, 3)])
def test_crowded(n, ny, nx, offset, cells):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from thruster_cx_code_b200 import _lib
    from thruster_cx_code_b200.physics_engine import accumulate_rho
    rng = np.random.default_rng(n)
    dx, cd = 0.0125, 1.602e-19 * 1e17 / 80.0
    if cells == "mixed":
        parts = [_cells(rng, k, ny, nx, c) for k, c in ((n // 3, 0), (n // 3, 30), (n - 2 * (n // 3), 0))]
        o = np.lexsort(parts[2][::-1])
        parts[2] = (parts[2][0][o], parts[2][1][o])
        iy, ix = (np.concatenate([p[k] for p in parts]) for k in (0, 1))
    else:
        iy, ix = _cells(rng, n, ny, nx, cells)
    dev = []
    for v in (ix, iy):
        t = torch.zeros(n + offset, dtype=torch.float32, device="cuda")[offset:]
        t.copy_(torch.from_numpy((v * dx).astype(np.float32)))
        dev.append(t)
    ref = (rng.integers(-3, 40, (ny, nx)) * np.float32(cd)).astype(np.float32)
    got = [torch.tensor(ref, device="cuda") for _ in range(2)]
    for sign in (1.0, -1.0, 1.0):
        accumulate_rho(*dev, got[0], n, dx, dx, nx, ny, sign * cd)
        _lib.check(_lib.load().pb_accumulate_rho_noalloc(
            *[C.c_void_p(t.data_ptr()) for t in (*dev, got[1])], n, dx, dx, nx, ny, sign * cd,
            torch.cuda.current_stream().cuda_stream), "noalloc")
        np.add.at(ref, (iy, ix), sign * cd)
    for g in got:
        np.testing.assert_array_equal(g.cpu().numpy().view(np.uint32), ref.view(np.uint32))
