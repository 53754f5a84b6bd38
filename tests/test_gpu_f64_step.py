"""The FP64 step kernel at the sizes where its numbering, division and read-back can go wrong: rows of
one and of a few nodes, rows one past a warp, blocks' remainders, walls on every axis, a body force and a
time-dependent mix of zero and non-zero non-equilibrium.  Bit for bit against the C restatement of the
reference's step."""
import numpy as np
import pytest

from fixtures import grid_order

pytestmark = pytest.mark.gpu
zl = pytest.importorskip("zllbm_b200")

WALL, PER = zl.BC_BOUNCE_BACK, zl.BC_PERIODIC


@pytest.mark.parametrize("coll", [zl.SRT, zl.MRT])
@pytest.mark.parametrize("force", [None, (3e-5, -1e-5, 2e-5)])
@pytest.mark.parametrize("n,bc", [((3, 3), (WALL,) * 4), ((33, 5), (WALL,) * 4), ((65, 9), (PER, PER, WALL, WALL)),
                                  ((129, 67), (WALL,) * 4), ((2, 3, 4), (WALL,) * 6), ((33, 4, 3), (WALL,) * 6),
                                  ((32, 5, 6), (PER, PER, WALL, WALL, PER, PER)), ((35, 3, 9), (PER,) * 6)])
def test_fp64_step_is_the_references(port, n, bc, coll, force):
    from oracle.port import LevelConfig
    dims = len(n)
    rng = np.random.default_rng(7)
    z3 = (0.0, 0.0, 0.0)
    vel = [z3] * 6
    if bc[3] == WALL:
        vel[3] = (0.05, 0.0, 0.02 if dims == 3 else 0.0)
    cfg = LevelConfig(dims=dims, n=tuple(n), collision=coll, nu=0.013, bc_kind=tuple(bc) + (0,) * (6 - len(bc)),
                      bc_vel=tuple(vel), force=force)
    # half of the box at rest (f = feq exactly there), the other half disturbed
    q = cfg.q
    f = np.tile(port.feq(dims, 1.0, [0.0] * dims), (int(np.prod(n)), 1))
    f[f.shape[0] // 2:] *= 1.0 + 0.02 * rng.standard_normal((f.shape[0] - f.shape[0] // 2, q))
    grid = f.reshape(tuple(reversed(n)) + (q,))
    for a in range(dims):  # a periodic axis stores its first plane twice
        if bc[2 * a] == PER:
            ax = dims - 1 - a
            np.moveaxis(grid, ax, 0)[-1] = np.moveaxis(grid, ax, 0)[0]
    codes = zl.box_codes(dims, [1] * dims, list(n))
    lin = grid_order(codes, dims, tuple(n))
    f0 = f[lin].copy()
    steps = 7
    port.run(cfg, f, f.copy(), steps)
    scfg = zl.SolverConfig(lattice=zl.D2Q9 if dims == 2 else zl.D3Q19, collision=coll, storage=zl.STORAGE_F64,
                           viscosity=cfg.nu, bc_kind=cfg.bc_kind, bc_velocity=cfg.bc_vel,
                           domain_min=(1, 1, 1 if dims == 3 else 0), domain_max=tuple(n) + (0,) * (3 - dims),
                           forcing=0 if force is None else 1, constant_force=force or z3)
    with zl.Context(scfg) as ctx:
        ctx.set_level_nodes(0, codes)
        ctx.set_populations(0, codes, f0)
        ctx.advance(steps)
        got = ctx.get_populations(0, codes)
    assert np.array_equal(got, f[lin]), np.abs(got - f[lin]).max()
