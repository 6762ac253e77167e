"""accumulate_rho beside the counts, rising with the square of the cells, from which the larger of the small
grids take several clusters."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,ny,nx", [(4_369_066, 160, 320), (4_369_067, 160, 320), (2_495_232, 129, 300),
                                     (2_496_151, 129, 300)])
def test_lines_by_cells(n, ny, nx):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from thruster_cx_code_b200.physics_engine import accumulate_rho
    rng = np.random.default_rng(n)
    dx, cd = 0.0125, 0.25
    iy, ix = rng.integers(1, ny - 1, n), rng.integers(1, nx - 1, n)
    x, y = (torch.from_numpy((v * dx).astype(np.float32)).cuda() for v in (ix, iy))
    rho = torch.zeros(ny, nx, device="cuda")
    accumulate_rho(x, y, rho, n, dx, dx, nx, ny, cd)  # whole quarters: the sum is exact
    ref = np.bincount(iy * nx + ix, minlength=ny * nx).reshape(ny, nx).astype(np.float32) * np.float32(cd)
    np.testing.assert_array_equal(rho.cpu().numpy(), ref)
