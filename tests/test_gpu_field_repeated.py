"""The joined field solve called again and again: calls whose Picard iterations need no linear solve, in
which its tables are never filled, and calls in which only some do, between ordinary ones; against the
general kernel (which a launch of fewer blocks than virtual blocks takes), bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

GRIDS2 = [dict(V=1000.0, t=0.38, gap=1.0, r=0.95, cham=0.0), dict(V=-200.0, t=1.0, gap=1.0, r=0.55, cham=0.0)]
PARAMS = dict(grids=GRIDS2, pitch_mm=3.75, Te_up=5.0, n0_plasma=1e17, Ti=0.1, sim_mode="Both")


def _calls(dx, blocks):
    from thruster_cx_code_b200 import _lib
    from thruster_cx_code_b200 import physics_engine as PE
    s = PE.DigitalTwinSimulator(seed=3)
    s.dx = s.dy = dx
    if blocks:
        _lib.check(s._libh.pb_sim_set_launch(s._h, 8, blocks), "set_launch")
    s.build_domain(PARAMS)
    r = np.random.default_rng(5)
    rho = (1e-3 * r.random((s.ny, s.nx)) * ~np.asarray(s.isBound)).astype(np.float32)
    out, inner = [], []
    for scale, calls in ((0.0, (60, 60, 60, 3, 1)), (1e-9, (5, 30)), (1.0, (5, 60, 60, 2)), (1.0 + 2.0 ** -20, (40, 1, 6))):
        s.rho = (np.float32(scale) * rho).astype(np.float32)
        for n in calls:
            s.recalc_poisson(iterations=n, params=PARAMS)
            out += [np.array(s.V), np.array(s.Ex), np.array(s.Ey), np.array(s.poisson_stats)]
            inner.append(s.poisson_stats[1])
    s.close()
    return out, np.diff(inner)


@pytest.mark.parametrize("dx", [0.035, 0.025, 0.0125])
def test_repeated_calls(dx):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    ref, inner = _calls(dx, 3)
    assert (inner == 0).any() and (inner > 0).any(), inner  # both kinds of call
    got, _ = _calls(dx, 0)
    for k, (a, b) in enumerate(zip(ref, got)):
        assert a.tobytes() == b.tobytes(), k
