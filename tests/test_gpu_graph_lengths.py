"""Captured step graphs of different lengths: calls of one step, of a few, of more than a graph holds and odd
ones, in any order, give the bits of single steps (the graph of a level is kept per layout, holds up to
sixteen steps, grows with the longest call so far, and the rest of a call is launched directly)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
zl = pytest.importorskip("zllbm_b200")
torch = pytest.importorskip("torch")

CALLS = [(2, 2, 40, 3, 1, 17, 16, 5), (33, 33, 1, 31), (1, 1, 64)]


def run(storage, calls, graph):
    n = (34, 12, 10)
    cfg = zl.SolverConfig(lattice=zl.D3Q19, collision=zl.SRT, storage=storage, viscosity=0.02,
                          bc_kind=(zl.BC_PERIODIC,) * 6, domain_min=(0, 0, 0), domain_max=n)
    g = torch.Generator(device="cuda")
    g.manual_seed(1)
    cells = n[0] * n[1] * n[2]
    rho = torch.ones(cells, device="cuda")
    u = (0.03 * torch.randn(cells, 3, generator=g, device="cuda")).contiguous()
    with zl.Context(cfg) as ctx:
        ctx.set_level_box(0, (0, 0, 0), n)
        torch.cuda.synchronize()
        ctx.set_equilibrium_dense(0, rho.data_ptr(), u.data_ptr())
        ctx.set_graph(graph)
        for k in calls:
            ctx.advance(k) if graph else [ctx.step_level(0) for _ in range(k)]
        ctx.get_macros_dense(0, rho.data_ptr(), u.data_ptr())
        ctx.synchronize()
    return rho.cpu().numpy(), u.cpu().numpy()


@pytest.mark.parametrize("storage", [zl.STORAGE_F32, zl.STORAGE_F16])
@pytest.mark.parametrize("calls", CALLS)
def test_graph_calls_equal_single_steps(storage, calls):
    a, b = run(storage, calls, True), run(storage, calls, False)
    assert np.array_equal(a[0], b[0]) and np.array_equal(a[1], b[1])
