"""Uploads to a simulator on another device than the thread's current one: the particles arrive and the
thread's device stays selected."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [5, 5000])
def test_upload_from_another_device(n):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available() or torch.cuda.device_count() < 2:
        pytest.skip("needs two CUDA devices")
    from thruster_cx_code_b200 import physics_engine as PE
    s = PE.DigitalTwinSimulator(device=1)
    torch.cuda.set_device(0)
    v = [np.arange(n, dtype=np.float32) + k for k in range(5)]
    for _ in range(2):  # storage made, then large enough already
        s.set_particles("ions", *v, sort=False)
        assert torch.cuda.current_device() == 0
    got = s._download_particles(0, n)
    for a, b in zip(got, v):
        np.testing.assert_array_equal(a, b)
    s.close()
    torch.cuda.set_device(0)
