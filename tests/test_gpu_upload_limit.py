"""A species holds its particles and a quarter more, counted in 32 bits: uploads whose storage does not fit
such a count are refused before anything is read."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_uploads_beyond_the_storage_are_refused():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from thruster_cx_code_b200 import _lib
    from thruster_cx_code_b200 import physics_engine as PE
    s = PE.DigitalTwinSimulator()
    v = [np.ones(4, np.float32) for _ in range(5)] + [np.zeros(4, np.uint8), np.zeros(4, np.uint32)]
    ptr = [a.ctypes.data_as(C.c_void_p) for a in v]
    top = C.c_int64(-1)
    for n in (1_717_983_442, 2_000_000_000, 2 ** 31 - 1):  # 1.25 n + 4096 reaches past int32
        for sp in (0, 1):
            assert s._libh.pb_sim_upload_particles(s._h, sp, n, *ptr, 0, 1, 0.1, 0.1, C.byref(top)) == 3
            assert s._libh.pb_sim_set_particles(s._h, sp, n, *ptr, 4) == 3
    assert top.value == -1
    s.close()
