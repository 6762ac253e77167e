"""set_particles, whose parts run as a pipeline: particles,
order, flags and next id against a stable argsort of the same cell keys, from pageable and
pinned arrays."""
import numpy as np
import pytest

from thruster_cx_code_b200 import workloads as W

pytestmark = pytest.mark.gpu
PIPE = 1 << 20


@pytest.fixture(scope="module")
def sim():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from thruster_cx_code_b200 import physics_engine as PE
    s = PE.DigitalTwinSimulator()
    s.build_domain(dict(grids=[dict(V=1000.0, t=0.38, gap=1.0, r=0.95, cham=0.0)], sim_mode="Both"))
    return s


@pytest.mark.parametrize("species", ["ions", "electrons"])
@pytest.mark.parametrize("n", [0, 1, 4097, PIPE - 1, PIPE, PIPE + 3])
@pytest.mark.parametrize("sort", [False, True])
@pytest.mark.parametrize("pinned", [False, True])
def test_upload(sim, species, n, sort, pinned):
    import torch
    r = np.random.default_rng(n + 7)
    a = [(r.random(n) * L).astype(np.float32) for L in (sim.Lx, sim.Ly)]
    a += [r.standard_normal(n).astype(np.float32) for _ in range(3)]
    ids = r.permutation(n).astype(np.uint32) + np.uint32(11)
    cex = (r.random(n) < 0.3).astype(np.uint8)
    if pinned and n:
        a = [torch.from_numpy(v).pin_memory().numpy() for v in a]
        ids = torch.from_numpy(ids.view(np.int32)).pin_memory().numpy().view(np.uint32)
    sp = int(species == "electrons")
    for next_id in (None, n + 1000):
        sim.set_particles(species, *a, is_cex=cex, ids=ids, sort=sort, next_id=next_id)
        top = n + 11 if n else 0
        assert (sim.next_e_id if sp else sim.next_ion_id) == (top if next_id is None else next_id)
        assert (sim.num_e if sp else sim.num_p) == n
        perm = np.arange(n)
        if sort:
            ix = np.clip(np.round(a[0] / np.float32(sim.dx)).astype(np.int64), 1, sim.nx - 2)
            iy = np.clip(np.round(a[1] / np.float32(sim.dy)).astype(np.int64), 1, sim.ny - 2)
            perm = np.argsort(iy * sim.nx + ix, kind="stable")
        got = sim._download_particles(sp, n)
        for g, v in zip(got[:5], a):
            np.testing.assert_array_equal(g.view(np.uint32), v[perm].view(np.uint32))
        np.testing.assert_array_equal(got[6], ids[perm])
        if sp == 0:
            np.testing.assert_array_equal(got[5], cex[perm].astype(bool))


def test_refused_sort_leaves_the_particles(sim):
    from thruster_cx_code_b200 import physics_engine as PE
    s = PE.DigitalTwinSimulator()
    v = np.ones(5, np.float32)
    with pytest.raises(RuntimeError):
        s.set_particles("ions", v, v, v, v, v, sort=True)   # no domain to sort by
    assert s.num_p == 5 and s.next_ion_id == 5
    np.testing.assert_array_equal(s._download_particles(0, 5)[0], v)
