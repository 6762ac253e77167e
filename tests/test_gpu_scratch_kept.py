"""The scratch of the largest packed push stays in the library's pool when the call is waited for
(memory given back at every synchronisation is mapped again by the next call, which takes longer
than the push), and pb_release_scratch gives it back."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ny,nx", [(2047, 2047), (1024, 4096), (513, 2049)])
def test_largest_push_keeps_its_scratch(ny, nx):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from thruster_cx_code_b200 import _lib
    from thruster_cx_code_b200.physics_engine import push_particles_boris
    n = max(600_000, (3 * ny * nx + 1) // 2)
    g = torch.Generator(device="cuda")
    g.manual_seed(ny)
    dx = 0.0125
    x = (nx - 1) * dx * torch.rand(n, generator=g, device="cuda")
    y = (ny - 1) * dx * torch.rand(n, generator=g, device="cuda")
    v = [torch.randn(n, generator=g, device="cuda") for _ in range(3)]
    F = [torch.randn(ny, nx, generator=g, device="cuda") for _ in range(2)]
    F += [torch.zeros(ny, nx, device="cuda") for _ in range(3)]
    assert _lib.load().pb_release_scratch() == 0
    push_particles_boris(x, y, *v, *F, n, dx, dx, nx, ny, 1e-12, 1e6)
    torch.cuda.synchronize()
    held = torch.cuda.mem_get_info()[0]
    assert _lib.load().pb_release_scratch() == 0
    assert torch.cuda.mem_get_info()[0] >= held + 80 * ny * nx
