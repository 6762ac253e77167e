"""The step's cooling and conduction for every value that an electrode mask of the C interface may
hold (any nonzero byte is an electrode cell): cells of an odd value conduct, cells of an even value
are cooled and do not.  The temperatures after one step against the same float32 operations in
NumPy, bit for bit."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
f32 = np.float32


@pytest.fixture(scope="module")
def PE():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from thruster_cx_code_b200 import physics_engine
    return physics_engine


def _expected(T, m, P):
    cf, T4, fx, fy = (f32(v) for v in (P.cooling_factor, P.T4_300, P.Fo_x, P.Fo_y))
    T = T.copy()
    cells = m != 0
    t = T[cells]
    T[cells] = t - cf * ((t.astype(np.float64) ** 2 * t.astype(np.float64) ** 2).astype(f32) - T4)
    on = (m & 1) == 1
    inside = np.zeros_like(on)
    inside[1:-1, 1:-1] = on[1:-1, 1:-1]
    for _ in range(P.sweeps):
        c = T
        n = [np.where(np.roll(on, s, a), np.roll(c, s, a), c) for s, a in ((1, 1), (-1, 1), (1, 0), (-1, 0))]
        tl, tr, td, tu = n
        c2 = f32(2.0) * c
        v = c + (fx * ((tl - c2) + tr) + fy * ((td - c2) + tu))
        T = np.where(inside, np.maximum(v, f32(300.0)), c)
    T[on] = np.maximum(T[on], f32(300.0))
    return T


@pytest.mark.parametrize("values", [(1,), (255,), (2,), (1, 2, 3, 128, 255)])
def test_cooling_and_conduction(PE, values):
    from thruster_cx_code_b200 import _lib
    params = dict(grids=[dict(V=1000.0, t=0.38, gap=1.0, r=0.95, cham=0.0)], sim_mode="Thermal")
    s = PE.DigitalTwinSimulator(seed=4)
    s.dx = s.dy = 0.05
    s.build_domain(params)
    rng = np.random.default_rng(11)
    ib = np.asarray(s.isBound).astype(bool)
    m = np.where(ib, rng.choice(np.array(values, np.uint8), ib.shape), np.uint8(0)).astype(np.uint8)
    s.Tmap = np.where(ib, rng.uniform(250.0, 900.0, ib.shape), 300.0).astype(f32)
    s._flush()
    _lib.check(s._libh.pb_sim_set_field(s._h, 6, m.ctypes.data_as(C.c_void_p), m.nbytes), "set_field")
    T0 = np.array(s.Tmap)
    P = s.step_params(params)
    assert P.thermal_on and P.sweeps > 0 and P.cooling_factor > 0
    s._upload_user_cs()
    R = _lib.StepReport()
    _lib.check(s._libh.pb_sim_step(s._h, C.byref(P), C.byref(R)), "pb_sim_step")
    got = np.empty(T0.shape, f32)
    _lib.check(s._libh.pb_sim_get_field(s._h, 4, got.ctypes.data_as(C.c_void_p), got.nbytes), "get_field")
    want = _expected(T0, m, P)
    np.testing.assert_array_equal(got.view(np.uint32), want.view(np.uint32))
    s.close()
