"""The module kernels with counts close to 2^31, where the index that ends a grid-stride loop lies
above it: deposit against the same deposit in smaller calls, push against its first and last particles
in calls of their own, conduction of an unmasked map against a copy, bit for bit."""
import pytest

pytestmark = pytest.mark.gpu
N = 2 ** 31 - 3


@pytest.fixture
def torch_cuda():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    torch.cuda.empty_cache()
    yield torch
    torch.cuda.empty_cache()


def _room(torch, nbytes):
    if torch.cuda.mem_get_info()[0] < nbytes + (4 << 30):
        pytest.skip("not enough device memory")


def _array(torch, n, offset, lo, hi, seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    t = torch.empty(n + offset, dtype=torch.float32, device="cuda")[offset:]
    return t.uniform_(lo, hi, generator=g)


@pytest.mark.parametrize("ny,nx,offset", [(257, 1025, 0), (257, 1025, 1), (65, 284, 0), (65, 284, 1)])
def test_deposit(torch_cuda, ny, nx, offset):
    torch = torch_cuda
    from thruster_cx_code_b200.physics_engine import accumulate_rho
    _room(torch, 8 * N)
    dx, cd = 0.0125, 1.602e-19 * 1e17 / 80.0
    x = _array(torch, N, offset, 0.0, (nx - 1) * dx, 1)
    y = _array(torch, N, offset, 0.0, (ny - 1) * dx, 2)
    got = [torch.zeros(ny, nx, device="cuda") for _ in range(2)]
    accumulate_rho(x, y, got[0], N, dx, dx, nx, ny, cd)
    for k in range(0, N, 1 << 28):
        px, py = x[k:k + (1 << 28)], y[k:k + (1 << 28)]
        accumulate_rho(px, py, got[1], px.numel(), dx, dx, nx, ny, cd)
    assert torch.equal(got[0].view(torch.int32), got[1].view(torch.int32))


@pytest.mark.parametrize("ny,nx,offset", [(257, 1025, 0), (257, 1025, 1), (2049, 2049, 0)])  # the last is not packed
def test_push(torch_cuda, ny, nx, offset):
    torch = torch_cuda
    from thruster_cx_code_b200.physics_engine import push_particles_boris
    _room(torch, 20 * N)
    dx, m = 0.0125, 300_001
    cols = [_array(torch, N, offset, 0.0, (L - 1) * dx, k) for k, L in enumerate((nx, ny))]
    cols += [_array(torch, N, offset, -1e5, 1e5, k) for k in (2, 3, 4)]
    F = [_array(torch, ny * nx, 0, -1e5, 1e5, 5 + k).view(ny, nx) for k in range(2)]
    F += [torch.zeros(ny, nx, device="cuda") for _ in range(3)]
    ends = [[c[a:b].clone() for c in cols] for a, b in ((0, m), (N - m, N))]
    push_particles_boris(*cols, *F, N, dx, dx, nx, ny, 2e-12, -1.9e9)
    for part, (a, b) in zip(ends, ((0, m), (N - m, N))):
        push_particles_boris(*part, *F, m, dx, dx, nx, ny, 2e-12, -1.9e9)
        for p, c in zip(part, cols):
            assert torch.equal(p.view(torch.int32), c[a:b].view(torch.int32))


@pytest.mark.parametrize("offset", [0, 1])
def test_conduction(torch_cuda, offset):
    torch = torch_cuda
    from thruster_cx_code_b200.physics_engine import thermal_conduction
    n = 46340
    _room(torch, 13 * n * n)
    T = _array(torch, n * n, offset, 250.0, 900.0, 9)
    out = torch.zeros(n * n + offset, dtype=torch.float32, device="cuda")[offset:]
    mask = torch.zeros(n * n + offset, dtype=torch.int32, device="cuda")[offset:]
    thermal_conduction(T, out, mask, n, n, 0.2, 0.2)
    assert torch.equal(T, out)
