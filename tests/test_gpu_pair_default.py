"""FP32 D3Q19 periodic boxes step two nodes per thread without being asked to.  Plain boxes: the bits of
the one-node kernel (which an explicit block shape selects), on rows that fill a warp's lanes and rows
that leave some idle.  Smagorinsky boxes, which take pairs whatever the block shape: FP64 storage to FP32
rounding."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
zl = pytest.importorskip("zllbm_b200")
torch = pytest.importorskip("torch")


def fields(n):
    g = torch.Generator(device="cuda")
    g.manual_seed(3)
    rho = 1.0 + 0.01 * torch.randn(n[0] * n[1] * n[2], generator=g, device="cuda")
    u = 0.03 * torch.randn(n[0] * n[1] * n[2], 3, generator=g, device="cuda")
    return rho.contiguous(), u.contiguous()


def run(n, coll, les, steps, block=None, storage=None):
    cfg = zl.SolverConfig(lattice=zl.D3Q19, collision=coll, storage=zl.STORAGE_F32 if storage is None else storage,
                          viscosity=0.002, bc_kind=(zl.BC_PERIODIC,) * 6, domain_min=(0, 0, 0), domain_max=n,
                          les=zl.LES_SMAGORINSKY if les else zl.LES_OFF, les_cs=0.1)
    rho, u = fields(n)
    out_r, out_u = torch.empty_like(rho), torch.empty_like(u)
    with zl.Context(cfg) as ctx:
        ctx.set_level_box(0, (0, 0, 0), n)
        if block:
            ctx.set_block(0, *block)
        torch.cuda.synchronize()
        ctx.set_equilibrium_dense(0, rho.data_ptr(), u.data_ptr())
        for _ in range(steps):
            ctx.step_level(0)
        ctx.get_macros_dense(0, out_r.data_ptr(), out_u.data_ptr())
        ctx.synchronize()
    return out_r.cpu().numpy(), out_u.cpu().numpy()


@pytest.mark.parametrize("coll", [zl.SRT, zl.MRT])
@pytest.mark.parametrize("n", [(128, 112, 110), (66, 161, 150)])
def test_default_kernel_has_the_one_node_kernels_bits(n, coll):
    a, b = run(n, coll, False, 3), run(n, coll, False, 3, (64, 2))
    assert np.array_equal(a[0], b[0]) and np.array_equal(a[1], b[1])


@pytest.mark.parametrize("coll", [zl.SRT, zl.MRT])
@pytest.mark.parametrize("n,block", [((96, 84, 80), None), ((66, 90, 91), (64, 4)), ((256, 48, 44), (32, 1))])
def test_smagorinsky_pairs_follow_fp64(n, coll, block):
    """Four steps against FP64 storage: FP32 rounding of the populations, a few 1e-7 of the velocity scale
    0.03 per step (tolerance 2e-6 absolute, 2e-6 on the density)."""
    a, ref = run(n, coll, True, 4, block), run(n, coll, True, 4, storage=zl.STORAGE_F64)
    assert np.abs(a[0] - ref[0]).max() <= 2e-6
    assert np.abs(a[1] - ref[1]).max() <= 2e-6
