"""The field solve with joined phases against the general kernel (which a launch of fewer blocks
than virtual blocks takes): the same potential, field and iteration counts, bit for bit, on odd
and even grids and for block counts that move the tiles and runs."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

GRIDS2 = [dict(V=1000.0, t=0.38, gap=1.0, r=0.95, cham=0.0), dict(V=-200.0, t=1.0, gap=1.0, r=0.55, cham=0.0)]
PARAMS = dict(grids=GRIDS2, pitch_mm=3.75, Te_up=5.0, n0_plasma=1e17, Ti=0.1, sim_mode="Both")


@pytest.fixture(scope="module")
def PE():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from thruster_cx_code_b200 import physics_engine
    return physics_engine


def _solve(PE, dx, blocks, geometry, max_coarse):
    from thruster_cx_code_b200 import _lib
    s = PE.DigitalTwinSimulator(seed=3, solver=dict(max_coarse=max_coarse))
    s.dx = s.dy = dx
    params = dict(PARAMS, geometry=geometry)
    if blocks:
        _lib.check(s._libh.pb_sim_set_launch(s._h, 8, blocks), "set_launch")
    s.build_domain(params)
    r = np.random.default_rng(5)
    out = [np.array(s.V)]
    for scale in (1.0, 3.0):
        s.rho = (scale * 1e-3 * r.random((s.ny, s.nx)) * ~np.asarray(s.isBound)).astype(np.float32)
        s.recalc_poisson(iterations=5, params=params)
        out += [np.array(s.V), np.array(s.Ex), np.array(s.Ey), np.array(s.poisson_stats)]
    shape = (s.ny, s.nx)
    s.close()
    return shape, out


@pytest.mark.parametrize("dx,geometry,max_coarse", [(0.025, "half_hole", 1536), (0.0311, "half_hole", 1536),
                                                    (0.019, "half_hole", 1536), (0.0125, "half_hole", 1536),
                                                    (0.01, "half_hole", 1536), (0.04, "one_hole", 1536),
                                                    (0.025, "half_hole", 200), (0.0125, "half_hole", 300),
                                                    (0.00625, "half_hole", 1536), (0.007, "half_hole", 300)])
def test_joined_phases_same_bits(PE, dx, geometry, max_coarse):
    shape, ref = _solve(PE, dx, 3, geometry, max_coarse)  # fewer blocks than virtual blocks
    for blocks in (0, 147, 61, 18):
        got_shape, got = _solve(PE, dx, blocks, geometry, max_coarse)
        assert got_shape == shape
        for a, b in zip(ref, got):
            assert a.tobytes() == b.tobytes(), (shape, blocks)
