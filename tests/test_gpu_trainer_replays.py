"""Training steps launched, replayed from a captured graph and captured without a replay, in any order: each
step's gradients and loss are those of a new trainer that launches one step from the same weights (the same
samples in the same tiles: FP32 atomic adds over at most 148 blocks in another order, 148 x 2^-24 of their
norm), and the weights follow Adam with those gradients.

The updates are restated in FP64 with the bias corrections rounded as the step rounds them: c2 = 1 - 0.999^t
in FP32 is off by up to 2^-24 / 0.001 = 6e-5 of itself, so an update (about lr) by less than 1e-4 lr, and a
weight (below 2) by another 2^-24 per step.  A captured step keeps the corrections of its capture."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
zl = pytest.importorskip("zllbm_b200")
torch = pytest.importorskip("torch")

LR = 1e-3
# L: a launched step, C: capture a step (not run), R: replay the last capture, 1 / 2: replay that capture
ORDERS = ["LCRLRL", "LCL", "LCLR", "CRRL", "LCRCRL", "LCLC1L2L1"]


def batch(n):
    g = torch.Generator(device="cuda")
    g.manual_seed(n)
    return torch.randn(n, 24, generator=g, device="cuda"), torch.rand(n, generator=g, device="cuda")


def one_launched_step(net, x, y, n):
    with zl.Trainer(net) as tr:
        torch.cuda.synchronize()
        tr.step(x.data_ptr(), y.data_ptr(), n, 0.0)
        return tr.gradients().flat()[:zl.MLP_TRAINABLE].astype(np.float64), tr.loss()


@pytest.mark.parametrize("n", [129, 128 * 297 + 77])
@pytest.mark.parametrize("order", ORDERS)
def test_steps_by_any_route(order, n):
    from zllbm_b200.hit import initial_net
    x, y = batch(n)
    side = torch.cuda.Stream()
    captured, calls = [], 0
    m = v = np.zeros(zl.MLP_TRAINABLE)
    with torch.cuda.stream(side), zl.Trainer(initial_net(5)) as tr:
        tr.set_stream(side.cuda_stream)
        torch.cuda.synchronize()
        for op in order:
            if op == "C":
                g = torch.cuda.CUDAGraph()
                with torch.cuda.graph(g, stream=side):
                    tr.step(x.data_ptr(), y.data_ptr(), n, LR)
                calls += 1
                captured.append((g, calls))
                continue
            before = tr.weights()
            if op == "L":
                tr.step(x.data_ptr(), y.data_ptr(), n, LR)
                calls += 1
                t = calls
            else:
                g, t = captured[-1 if op == "R" else int(op) - 1]
                g.replay()
            grad, loss = tr.gradients().flat()[:zl.MLP_TRAINABLE].astype(np.float64), tr.loss()
            ref, ref_loss = one_launched_step(before, x, y, n)
            assert np.linalg.norm(grad - ref) <= 148 * 2.0 ** -24 * np.linalg.norm(ref)
            assert np.isclose(loss, ref_loss, rtol=148 * 2.0 ** -24)
            m, v = 0.9 * m + 0.1 * grad, 0.999 * v + 0.001 * grad * grad
            c1, c2 = (float(np.float32(1) - np.float32(b) ** np.float32(t)) for b in (0.9, 0.999))
            w = before.flat()[:zl.MLP_TRAINABLE].astype(np.float64)
            expect = w - LR * (m / c1) / (np.sqrt(v / c2) + 1e-8)
            now = tr.weights().flat()[:zl.MLP_TRAINABLE]
            assert np.abs(w).max() < 2.0
            assert np.abs(now - expect).max() <= 1e-4 * LR + 2.0 ** -24
