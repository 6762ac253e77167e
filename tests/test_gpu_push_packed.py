"""pb_push_particles_boris packs the field corners first for large calls; smaller calls gather
from the arrays.  Both must give the same bits: one large call against the same particles
pushed in calls too small for the packed path, at counts around the dispatch line and the
four-particle vectors, on small and ragged grids, for arrays that do and do not start on a
16-byte boundary, for B zero, negative zero (a B field with its own signed zeros), ordinary and
non-finite, with particles outside the grid, on nodes and non-finite."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CHUNK = 50_000  # below the packed path's smallest call


@pytest.fixture(scope="module")
def torch_cuda():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return torch


def _case(torch, n, ny, nx, bkind, offset, seed):
    rng = np.random.default_rng(seed)
    dx = 0.0125
    Lx, Ly = (nx - 1) * dx, (ny - 1) * dx
    x = rng.uniform(-0.05 * Lx, 1.05 * Lx, n)
    y = rng.uniform(-0.05 * Ly, 1.05 * Ly, n)
    x[: n // 50] = dx * rng.integers(0, nx, n // 50)  # on nodes
    v = [1e5 * rng.standard_normal(n) for _ in range(3)]
    cols = [c.astype(np.float32) for c in (x, y, *v)]
    cols[2][5:9] = 0.0
    cols[3][7:12] = -0.0
    for c, bad in zip(cols, (np.nan, np.inf, -np.inf, np.nan, np.inf)):
        c[13:16] = bad
    dev = torch.device("cuda", 0)
    out = []
    for c in cols:
        t = torch.zeros(n + offset, dtype=torch.float32, device=dev)[offset:]
        t.copy_(torch.from_numpy(c))
        out.append(t)
    E = [torch.tensor((1e6 * rng.standard_normal((ny, nx))).astype(np.float32), device=dev) for _ in range(2)]
    B = [torch.zeros((ny, nx), dtype=torch.float32, device=dev) for _ in range(3)]
    if bkind == "negzero":
        B[1].fill_(-0.0)
    elif bkind == "one":
        B[2][ny - 1, nx - 1] = 0.3  # a single node, in the last row and column
    elif bkind == "field":
        B = [torch.tensor(rng.uniform(-0.2, 0.2, (ny, nx)).astype(np.float32), device=dev) for _ in range(3)]
    elif bkind == "nan":
        B[0][ny // 2, nx // 2] = float("nan")
        B[1][0, 0] = float("inf")
    return out, E, B, dx


@pytest.mark.parametrize("bkind", ["zero", "negzero", "one", "field", "nan"])
@pytest.mark.parametrize("n,ny,nx,offset", [(599_999, 65, 284, 0), (600_000, 65, 284, 0), (600_003, 2, 2, 0),
                                            (631_071, 33, 67, 1), (700_001, 130, 568, 0), (1_600_002, 513, 2049, 0)])
def test_packed_push_equals_direct(torch_cuda, n, ny, nx, offset, bkind):
    torch = torch_cuda
    from thruster_cx_code_b200.physics_engine import push_particles_boris
    big, E, B, dx = _case(torch, n, ny, nx, bkind, offset, n)
    small = [c.clone() for c in big]
    for _ in range(2):
        push_particles_boris(*big, *E, *B, n, dx, dx, nx, ny, 2e-12, -1.9e9)
        for k in range(0, n, CHUNK):
            part = [c[k:k + CHUNK] for c in small]
            push_particles_boris(*part, *E, *B, part[0].numel(), dx, dx, nx, ny, 2e-12, -1.9e9)
    torch.cuda.synchronize()
    for a, b in zip(big, small):
        nan = torch.isnan(a)
        assert torch.equal(nan, torch.isnan(b))
        assert torch.equal(a[~nan].view(torch.int32), b[~nan].view(torch.int32))


def test_scratch_release(torch_cuda):
    torch = torch_cuda
    from thruster_cx_code_b200 import _lib
    from thruster_cx_code_b200.physics_engine import push_particles_boris
    cols, E, B, dx = _case(torch, 1_700_000, 513, 2049, "field", 0, 1)
    push_particles_boris(*cols, *E, *B, 1_700_000, dx, dx, 2049, 513, 2e-12, -1.9e9)
    torch.cuda.synchronize()
    held = torch.cuda.mem_get_info()[0]
    assert _lib.load().pb_release_scratch() == 0
    assert torch.cuda.mem_get_info()[0] >= held + 513 * 2049 * 80
