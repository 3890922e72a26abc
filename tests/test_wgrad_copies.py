"""The buffers of the copies that weight gradients are formed from hold those of
every layer, whatever the widths of the levels.
"""

import pytest

from sunlightlb_gb300 import warmstart as WS


class Layout(WS.UNet):
    """A network's layers and training buffers, without a GPU."""

    def __init__(self, D, H, W, batch, widths):
        self.torch = pytest.importorskip("torch")
        self.D, self.H, self.W, self.B, self.widths = D, H, W, batch, widths
        self.dev, self.t, self.grad, self.clip_state = "meta", 0, None, None
        w0, w1, w2, w3 = widths
        couts = [(0, WS.IN_CH, w0), (0, w0, w0), (1, w0, w1), (1, w1, w1), (2, w1, w2), (2, w2, w2), (3, w2, w3), (3, w3, w3),
                 (2, w3 + w2, w2), (1, w2 + w1, w1), (0, w1 + w0, w0), (0, w0, WS.OUT_CH)]
        self.layers = [(f"l{i}", lv, cin, cout) for i, (lv, cin, cout) in enumerate(couts)]
        self.buf_spec = {"C0": (0, w1 + w0), "C1": (1, w2 + w1), "C2": (2, w3 + w2), "IN": (0, WS.IN_CH), "B3": (3, w3)}
        self.params = {n: {"w": self.torch.zeros(1), "b": self.torch.zeros(1)} for n, *_ in self.layers}


@pytest.mark.parametrize("widths", [(32, 64, 128, 256), (128, 32, 32, 32), (32, 32, 32, 256), (64, 128, 32, 32), (32, 32, 32, 32)])
def test_buffers_hold_every_layer(widths):
    net = Layout(32, 32, 64, 2, widths)
    net._alloc_grads()
    for _, lv, cin, cout in net.layers:
        d, h, w = net.dims(lv)
        Wp, ps = WS.flat_geometry(d, h, w)
        copies = 1 if cout <= 128 else 3
        assert net.cm_x.numel() >= cin * net.B * ps
        assert net.cm_g.numel() >= copies * cout * net.B * ps, (widths, lv, cout)
