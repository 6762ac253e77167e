"""Sputter breaks between steps taken one at a time through the C interface, each with its report and
without a new domain after a break: the hierarchy is rebuilt on the device before the next field solve,
as inside one pb_sim_run, and once the report after a rebuild names no broken cell the rebuild's launch
is left out again, for plain steps and for replayed step graphs.  Breaks are planted before step 0
and, under the same parameters, before step 8, so that the second rebuild step replays the first one's
graph."""
import ctypes as C

import numpy as np
import pytest

from thruster_cx_code_b200 import workloads as W

pytestmark = pytest.mark.gpu
K, AGAIN = 16, 8


@pytest.fixture(scope="module")
def lib():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from thruster_cx_code_b200 import _lib
    return _lib


def _sim():
    s, p = W.make_sweep_sim(W.sweep_point(np.random.default_rng(7), 0, grids=("64x256",), n_range=(150000, 150001)))
    p = dict(p, Thresh=1e9)
    s._flush()
    s._upload_user_cs()
    ib = np.asarray(s.isBound).astype(bool)
    col = np.arange(s.nx)[None, :] * s.dx
    left, right = np.zeros_like(ib), np.zeros_like(ib)
    left[:, 1:], right[:, :-1] = ~ib[:, :-1], ~ib[:, 1:]
    faces = [ib & left & (col < s.grid_x_starts[1]), ib & right & (col >= s.grid_x_starts[1])]
    steps = []
    for k in range(K):
        s.iteration = k
        steps.append(s.step_params(p))
    return s, faces, steps


def _plant(lib, s, face):
    d = np.where(face, 2e9, 0.0)
    lib.check(lib.load().pb_sim_set_field(s._h, 5, d.ctypes.data_as(C.c_void_p), d.nbytes), "set_field")


def _state(lib, s):
    h = lib.load()
    out = []
    for fid, dt in ((0, np.float64), (1, np.float32), (6, np.uint8), (12, np.uint8), (13, np.float32)):
        a = np.empty((s.ny, s.nx), dt)
        lib.check(h.pb_sim_get_field(s._h, fid, a.ctypes.data_as(C.c_void_p), a.nbytes), "get_field")
        out.append(a.tobytes())
    n = [C.c_int32(), C.c_int32()]
    ids = [C.c_uint32(), C.c_uint32()]
    lib.check(h.pb_sim_counts(s._h, *[C.byref(v) for v in n + ids]), "counts")
    for sp in (0, 1):
        out += [None if a is None else a.tobytes() for a in s._download_particles(sp, n[sp].value)]
    d = C.c_uint64()
    lib.check(h.pb_sim_operator_digest(s._h, C.byref(d)), "digest")
    return out + [d.value]


def test_steps_rebuild_and_leave_out(lib):
    h = lib.load()
    ref, faces, steps = _sim()
    for lo, hi, face in ((0, AGAIN, faces[0]), (AGAIN, K, faces[1])):
        _plant(lib, ref, face)
        P = (lib.StepParams * (hi - lo))(*steps[lo:hi])
        R = (lib.StepReport * (hi - lo))()
        lib.check(h.pb_sim_run(ref._h, P, hi - lo, R), "pb_sim_run")
        assert R[0].broken >= face.sum() > 0 and not any(r.broken for r in R[1:])
    want = _state(lib, ref)
    solves = [bool(q.do_poisson) for q in steps]
    for graphs in (0, 1):
        s, _, steps = _sim()
        lib.check(h.pb_sim_set_graphs(s._h, graphs), "set_graphs")
        launches = []
        for k in range(K):
            if k in (0, AGAIN):
                _plant(lib, s, faces[k == AGAIN])
            R = lib.StepReport()
            lib.check(h.pb_sim_step(s._h, C.byref(steps[k]), C.byref(R)), "pb_sim_step")
            assert (R.broken > 0) == (k in (0, AGAIN))
            prof = (C.c_double * 16)()
            lib.check(h.pb_sim_timing(s._h, prof), "pb_sim_timing")
            launches.append(int(prof[8]))
        assert _state(lib, s) == want, graphs
        if graphs:
            g = (C.c_int64 * 4)()
            lib.check(h.pb_sim_graph_stats(s._h, g), "graph_stats")
            assert g[1] >= 4 and g[3] == 0, list(g)
        # one launch more in the first field solve after a break, and in that one only
        first = [k for b in (0, AGAIN) for k in [next(j for j in range(b + 1, K) if solves[j])]]
        plain = [launches[k] for k in range(1, K) if solves[k] and k not in first]
        assert len(plain) >= 4 and set(plain) == {plain[0]}, launches
        assert [launches[k] for k in first] == [plain[0] + 1] * 2, launches
        s.close()
    ref.close()
