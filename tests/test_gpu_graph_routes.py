"""zl_advance by every route of its graphs gives the bits of single steps: launched, replayed in pairs, replayed
in a long graph that is captured later and grows, from both layouts, and after a change of the block shape (all
graphs captured anew).  A periodic box, whose step is one launch, and a box whose faces are passes in order
behind the step (pairs are kept beside the long graph)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
zl = pytest.importorskip("zllbm_b200")
torch = pytest.importorskip("torch")

CALLS = [8, 3, 40, 60, 10, 9, 14, 1, 14, 2, 16, 7, "block", 5, 260, 31, 1, 260, 15]


def run(ordered, graph):
    n = (34, 12, 10)
    wall, rest = zl.BC_BOUNCE_BACK, (0.0, 0.0, 0.0)
    inflow = (0.03, 0.0, 0.0)
    if ordered:
        cfg = zl.SolverConfig(lattice=zl.D3Q19, collision=zl.SRT, storage=zl.STORAGE_F32, viscosity=0.05,
                              bc_kind=(zl.BC_NONEQ_EXTRAPOLATION, zl.BC_CONVECTIVE_OUTFLOW) + (wall,) * 4,
                              bc_velocity=(inflow, inflow) + (rest,) * 4, domain_min=(0, 0, 0),
                              domain_max=tuple(k - 1 for k in n))
    else:
        cfg = zl.SolverConfig(lattice=zl.D3Q19, collision=zl.SRT, storage=zl.STORAGE_F32, viscosity=0.05,
                              bc_kind=(zl.BC_PERIODIC,) * 6, domain_min=(0, 0, 0), domain_max=n)
    g = torch.Generator(device="cuda")
    g.manual_seed(1)
    cells = n[0] * n[1] * n[2]
    rho = torch.ones(cells, device="cuda")
    u = (0.02 * torch.randn(cells, 3, generator=g, device="cuda")).contiguous()
    states = []
    with zl.Context(cfg) as ctx:
        ctx.set_level_box(0, (0, 0, 0), n)
        torch.cuda.synchronize()
        ctx.set_equilibrium_dense(0, rho.data_ptr(), u.data_ptr())
        ctx.set_graph(graph)
        for k in CALLS:
            if k == "block":
                ctx.set_block(0, 64, 2)
                continue
            ctx.advance(k) if graph else [ctx.step_level(0) for _ in range(k)]
            ctx.get_macros_dense(0, rho.data_ptr(), u.data_ptr())
            ctx.synchronize()
            states.append((rho.cpu().numpy(), u.cpu().numpy()))
    return states


@pytest.mark.parametrize("ordered", [False, True])
def test_every_route_equals_single_steps(ordered):
    a, b = run(ordered, True), run(ordered, False)
    assert np.isfinite(b[-1][0]).all()
    for (r0, u0), (r1, u1) in zip(a, b):
        assert np.array_equal(r0, r1) and np.array_equal(u0, u1)
