"""The training workload of the profiling cases is timed on the stream its steps run on."""
import pytest

pytestmark = pytest.mark.gpu
zl = pytest.importorskip("zllbm_b200")


def test_train_case_steps_on_the_timed_stream(monkeypatch):
    from zllbm_b200 import kernel_cases
    used, timed = [], []
    set_stream, events = zl.Trainer.set_stream, kernel_cases._events
    monkeypatch.setattr(zl.Trainer, "set_stream", lambda tr, s: (used.append(s), set_stream(tr, s)))
    monkeypatch.setattr(kernel_cases, "_events", lambda s, *a, **k: (timed.append(s), events(s, *a, **k))[1])
    rate = kernel_cases.train_case(4096, steps=2)
    # stream 0 would leave the trainer on a stream of its own, which events on the default stream do not see
    assert rate > 0.0 and used == timed and used[0] != 0
