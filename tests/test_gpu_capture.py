"""The module functions inside torch CUDA graphs: captured alone, in a chain, and behind the join of
another stream's work, at sizes of each of their routes, and replayed on new inputs, against the same
calls without a graph, bit for bit."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def torch_cuda():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return torch


def _state(torch, n, ny, nx, seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    dx = 0.0125
    r = [torch.rand(n, generator=g, device="cuda") for _ in range(2)]
    return dict(x=r[0] * ((nx - 1) * dx), y=r[1] * ((ny - 1) * dx),
                v=[1e5 * torch.randn(n, generator=g, device="cuda") for _ in range(3)],
                E=[1e5 * torch.randn(ny, nx, generator=g, device="cuda") for _ in range(2)],
                B=[0.1 * torch.rand(ny, nx, generator=g, device="cuda") for _ in range(3)],
                rho=torch.zeros(ny, nx, device="cuda"),
                T=[300.0 + 500.0 * torch.rand(ny, nx, generator=g, device="cuda") for _ in range(2)],
                mask=(torch.rand(ny, nx, generator=g, device="cuda") < 0.7).int())


def _tensors(s):
    return [s["x"], s["y"], *s["v"], s["rho"], *s["T"]]


def _work(torch, s, n, ny, nx, side):
    """Deposit, two conduction sweeps (on the stream side, if any), push, two sweeps behind their join,
    deposit."""
    from thruster_cx_code_b200.physics_engine import accumulate_rho, push_particles_boris, thermal_conduction
    dx = 0.0125
    here = torch.cuda.current_stream()
    side = side or here

    def sweeps():
        thermal_conduction(s["T"][0], s["T"][1], s["mask"], nx, ny, 0.2, 0.15)
        thermal_conduction(s["T"][1], s["T"][0], s["mask"], nx, ny, 0.2, 0.15)

    s["rho"].zero_()
    accumulate_rho(s["x"], s["y"], s["rho"], n, dx, dx, nx, ny, 0.25)
    if side is not here:
        side.wait_stream(here)
    with torch.cuda.stream(side):
        sweeps()
    push_particles_boris(s["x"], s["y"], *s["v"], *s["E"], *s["B"], n, dx, dx, nx, ny, 2e-12, -1.9e9)
    if side is not here:
        here.wait_stream(side)
    sweeps()
    accumulate_rho(s["x"], s["y"], s["rho"], n, dx, dx, nx, ny, -0.25)


@pytest.mark.parametrize("forked", [False, True])
@pytest.mark.parametrize("n,ny,nx", [(1000, 65, 284), (99_999, 160, 320), (400_001, 65, 284), (1_000_003, 65, 284),
                                     (700_000, 257, 1025)])
def test_captured_calls(torch_cuda, n, ny, nx, forked):
    torch = torch_cuda
    s, ref = _state(torch, n, ny, nx, 1), _state(torch, n, ny, nx, 1)
    side = torch.cuda.Stream() if forked else None
    start = [t.clone() for t in _tensors(s)]
    _work(torch, s, n, ny, nx, side)  # the libraries' set-up, outside the capture
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        _work(torch, s, n, ny, nx, side)
    for again in (1, 2):  # the same graph on the first inputs and on others
        new = start if again == 1 else [t.clone() for t in _tensors(_state(torch, n, ny, nx, 7))]
        for state in (s, ref):
            for t, v in zip(_tensors(state), new):
                t.copy_(v)
        for _ in range(2):
            graph.replay()
            _work(torch, ref, n, ny, nx, None)
        torch.cuda.synchronize()
        for a, b in zip(_tensors(s), _tensors(ref)):
            assert torch.equal(a.view(torch.int32), b.view(torch.int32))
    del graph
