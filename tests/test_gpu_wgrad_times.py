"""The weight-gradient times of the layers (warmstart.wgrad_layer_times) are of
the kernels a training step launches for them.
"""

import pytest

from sunlightlb_gb300 import warmstart as WS

pytestmark = pytest.mark.gpu


class Recorder:
    """Kernels that notes (entry point, cin, cout) of every weight gradient."""

    def __init__(self, kernels, seen):
        self.kernels, self.seen = kernels, seen

    def __getattr__(self, name):
        fn = getattr(self.kernels, name)
        if not name.startswith("tc_wgrad") or name == "tc_wgrad_splits":
            return fn

        def call(*a):
            self.seen.add((name,) + tuple(a[-7:-5]))  # cin, cout, workspace, floats, splits, result, stream
            return fn(*a)
        return call


def test_times_are_of_the_kernels_of_training(gpu, monkeypatch):
    torch = pytest.importorskip("torch")
    widths, make = (32, 64, 128, 256), WS.Kernels
    trained, timed = set(), set()
    monkeypatch.setattr(WS, "Kernels", lambda dll: Recorder(make(dll), trained))
    net = WS.UNet(gpu, 32, 32, 64, batch=1, widths=widths, seed=3)
    net.encode(torch.zeros(1, 32, 32, 64, device="cuda", dtype=torch.uint8))
    net.forward()
    net.loss_and_backward(torch.zeros(1, 32, 32, 64, 4, device="cuda"))
    monkeypatch.setattr(WS, "Kernels", lambda dll: Recorder(make(dll), timed))
    rows = WS.wgrad_layer_times(gpu, 32, 1, widths=widths, reps=2)
    assert timed == trained and len(timed) == len({r[1:3] for r in rows})
    assert all(r[4] > 0 for r in rows)
