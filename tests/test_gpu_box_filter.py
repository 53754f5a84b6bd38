"""The box filter's two kernels against a float64 block mean of the level's own fields: factors that divide
a warp (one and two sub-warp columns, a row that is not a multiple of 32, a factor of a whole row) and one
that does not.  Tolerance: the worst-case FP32 rounding of a thread's sequential sum (factor^2 or factor^3
terms), of the adds that follow it and of the values themselves, times the field's scale."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
zl = pytest.importorskip("zllbm_b200")
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("storage", [zl.STORAGE_F32, zl.STORAGE_F16])
@pytest.mark.parametrize("n,factor", [((32, 4, 4), 2), ((40, 8, 16), 4), ((72, 8, 8), 8), ((64, 16, 16), 16),
                                      ((36, 6, 9), 3), ((33, 5, 7), 1)])
@pytest.mark.parametrize("steps", [0, 1])
def test_filter_is_the_block_mean(n, factor, storage, steps):
    cfg = zl.SolverConfig(lattice=zl.D3Q19, collision=zl.SRT, storage=storage, viscosity=0.01,
                          bc_kind=(zl.BC_PERIODIC,) * 6, domain_min=(0, 0, 0), domain_max=n)
    g = torch.Generator(device="cuda")
    g.manual_seed(5)
    cells = n[0] * n[1] * n[2]
    rho = (1.0 + 0.02 * torch.randn(cells, generator=g, device="cuda")).contiguous()
    u = (0.05 * torch.randn(cells, 3, generator=g, device="cuda")).contiguous()
    m = [v // factor for v in n]
    out = torch.empty(m[0] * m[1] * m[2], 29, device="cuda")
    with zl.Context(cfg) as ctx:
        ctx.set_level_box(0, (0, 0, 0), n)
        torch.cuda.synchronize()
        ctx.set_equilibrium_dense(0, rho.data_ptr(), u.data_ptr())
        for _ in range(steps):
            ctx.step_level(0)
        ctx.get_macros_dense(0, rho.data_ptr(), u.data_ptr())
        ctx.filter_level(0, factor, out.data_ptr())
        ctx.synchronize()
    r = rho.double().cpu().numpy().reshape(n[::-1])
    v = u.double().cpu().numpy().reshape(n[::-1] + (3,))
    mean = lambda a: a.reshape(m[2], factor, m[1], factor, m[0], factor).mean(axis=(1, 3, 5)).ravel()
    got = out.double().cpu().numpy()
    terms = (factor ** 3 if factor & (factor - 1) else factor ** 2 + 5) + 8
    tol = terms * 2.0 ** -24
    assert np.abs(got[:, 0] - mean(r)).max() <= tol * r.max()
    for a in range(3):
        assert np.abs(got[:, 1 + a] - mean(v[..., a])).max() <= tol * np.abs(v).max()
        assert np.abs(got[:, 4 + a] - mean(v[..., a] ** 2)).max() <= tol * (v ** 2).max()
    # f - feq carries no mass: the 19 columns sum to zero
    assert np.abs(got[:, 10:].sum(axis=1)).max() <= tol
