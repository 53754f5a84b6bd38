"""Smagorinsky boxes in FP32: the caller chooses between one and two nodes per thread (zl_set_block), and the
choice changes no bit; the autotuner's choice can be set again; what the pair kernel cannot take is refused."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
zl = pytest.importorskip("zllbm_b200")
torch = pytest.importorskip("torch")


def config(n, coll, storage=None, les=True, forcing=None):
    return zl.SolverConfig(lattice=zl.D3Q19, collision=coll, storage=zl.STORAGE_F32 if storage is None else storage,
                           viscosity=0.002, bc_kind=(zl.BC_PERIODIC,) * 6, domain_min=(0, 0, 0), domain_max=n,
                           les=zl.LES_SMAGORINSKY if les else zl.LES_OFF, les_cs=0.1, forcing=1 if forcing is not None else 0,
                           constant_force=(forcing or 0.0, 0.0, 0.0))


def run(n, coll, choose):
    g = torch.Generator(device="cuda")
    g.manual_seed(3)
    cells = n[0] * n[1] * n[2]
    rho = 1.0 + 0.01 * torch.randn(cells, generator=g, device="cuda")
    u = 0.03 * torch.randn(cells, 3, generator=g, device="cuda")
    with zl.Context(config(n, coll)) as ctx:
        ctx.set_level_box(0, (0, 0, 0), n)
        torch.cuda.synchronize()
        ctx.set_equilibrium_dense(0, rho.data_ptr(), u.data_ptr())
        choose(ctx)
        for _ in range(3):
            ctx.step_level(0)
        ctx.get_macros_dense(0, rho.data_ptr(), u.data_ptr())
        ctx.synchronize()
    return rho.cpu().numpy(), u.cpu().numpy()


def tuned(ctx):
    x, y = ctx.autotune(0, trials=2)
    ctx.set_block(0, x, y)


@pytest.mark.parametrize("coll", [zl.SRT, zl.MRT])
@pytest.mark.parametrize("n", [(66, 90, 91), (24, 20, 18), (128, 70, 60)])
def test_every_shape_gives_the_same_bits(n, coll):
    ref = run(n, coll, lambda ctx: ctx.set_block(0, 64, 2))
    assert np.isfinite(ref[1]).all()
    for choose in (lambda ctx: None, lambda ctx: ctx.set_block(0, -64, 2), lambda ctx: ctx.set_block(0, -32, 8),
                   lambda ctx: ctx.set_block(0, 32, 4), tuned):
        a = run(n, coll, choose)
        assert np.array_equal(a[0], ref[0]) and np.array_equal(a[1], ref[1])


@pytest.mark.parametrize("n,storage,forcing", [((65, 20, 20), zl.STORAGE_F32, None),
                                               ((64, 20, 20), zl.STORAGE_F64, None),
                                               ((64, 20, 20), zl.STORAGE_F16, None),
                                               ((64, 20, 20), zl.STORAGE_F32, 1e-6)])
def test_pairs_are_refused_where_they_do_not_apply(n, storage, forcing):
    with zl.Context(config(n, zl.SRT, storage, forcing=forcing)) as ctx:
        ctx.set_level_box(0, (0, 0, 0), n)
        with pytest.raises(zl.ZlError):
            ctx.set_block(0, -64, 1)
        ctx.set_block(0, 64, 1)


def test_a_level_that_a_body_makes_forced_leaves_the_pairs():
    """Pairs are chosen while the level has no force; its immersed boundary then takes the one-node kernel for
    every node."""
    n = (64, 20, 18)
    out = []
    for block in (None, (-64, 1)):
        g = torch.Generator(device="cuda")
        g.manual_seed(4)
        rho = torch.ones(n[0] * n[1] * n[2], device="cuda")
        u = 0.02 * torch.randn(n[0] * n[1] * n[2], 3, generator=g, device="cuda")
        with zl.Context(config(n, zl.SRT, forcing=0.0)) as ctx:
            ctx.set_level_box(0, (0, 0, 0), n)
            torch.cuda.synchronize()
            ctx.set_equilibrium_dense(0, rho.data_ptr(), u.data_ptr())
            if block:
                ctx.set_block(0, *block)
            t = np.linspace(0.0, 2.0 * np.pi, 12, endpoint=False)
            xyz = np.stack([20.0 + 3.0 * np.cos(t), 10.0 + 3.0 * np.sin(t), np.full(12, 9.0)], axis=1)
            ctx.ib_set_vertices(0, xyz, np.zeros_like(xyz), np.ones(12))
            for _ in range(3):
                ctx.step_level(0)
            ctx.get_macros_dense(0, rho.data_ptr(), u.data_ptr())
            ctx.synchronize()
        out.append((rho.cpu().numpy(), u.cpu().numpy()))
    assert np.abs(out[0][1]).max() > 0.01
    assert np.array_equal(out[0][0], out[1][0]) and np.array_equal(out[0][1], out[1][1])
