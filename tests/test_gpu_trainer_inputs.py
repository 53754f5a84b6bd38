"""The training step on feature arrays that are not 16-byte aligned (read element by element instead of in
16-byte pieces), on batches of one tile, of two, of one more than the GPU takes at once and of a partial
last tile, and inside a captured CUDA graph that is replayed: the gradients of the aligned, launched step.
The same samples in the same tiles: the gradients differ by the order of FP32 atomic adds over at most 148
blocks, 148 x 2^-24 of their norm."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
zl = pytest.importorskip("zllbm_b200")
torch = pytest.importorskip("torch")


def data(n):
    g = torch.Generator(device="cuda")
    g.manual_seed(n)
    x = torch.randn(n * 24 + 4, generator=g, device="cuda")
    return x, torch.rand(n, generator=g, device="cuda")


def gradients(x, y, n, graph=False):
    from zllbm_b200.hit import initial_net
    side = torch.cuda.Stream()
    with torch.cuda.stream(side), zl.Trainer(initial_net(5)) as tr:
        tr.set_stream(side.cuda_stream)
        torch.cuda.synchronize()
        if graph:
            g = torch.cuda.CUDAGraph()
            with torch.cuda.graph(g, stream=side):
                tr.step(x.data_ptr(), y.data_ptr(), n, 0.0)
            for _ in range(3):
                g.replay()
            torch.cuda.synchronize()
        else:
            for _ in range(3):
                tr.step(x.data_ptr(), y.data_ptr(), n, 0.0)
        return tr.gradients().flat()[:zl.MLP_TRAINABLE].astype(np.float64), tr.loss() if not graph else None


@pytest.mark.parametrize("n", [1, 128, 129, 128 * 148 + 1, 128 * 297 + 77])
def test_unaligned_features_and_captured_steps(n):
    x, y = data(n)
    ref, loss = gradients(x[:n * 24], y, n)
    moved = torch.empty_like(x)
    moved[1:1 + n * 24] = x[:n * 24]
    odd, odd_loss = gradients(moved[1:1 + n * 24], y, n)
    cap, _ = gradients(x[:n * 24], y, n, graph=True)
    tol = 148 * 2.0 ** -24 * np.linalg.norm(ref)
    assert np.isfinite(loss) and np.isclose(odd_loss, loss, rtol=148 * 2.0 ** -24)
    assert np.linalg.norm(odd - ref) <= tol
    assert np.linalg.norm(cap - ref) <= tol
