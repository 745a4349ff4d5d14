"""sdem_sg_set_tensor_path governs the network's forward and training passes: with
0 no tcgen05 kernel is asked for, and the results are the same bits."""
import numpy as np
import pytest
import torch

from sdem_gb300 import build, surrogate as sg

pytestmark = pytest.mark.gpu
DEV = "cuda"


class Calls:
    """The library, with the names of the functions that were called."""

    def __init__(self, lib):
        self.lib, self.names = lib, []

    def __getattr__(self, name):
        self.names.append(name)
        return getattr(self.lib, name)


def test_forward_and_training():
    build.build()
    lib = sg.load()
    rng = np.random.default_rng(4)
    n, d = 800, 1.2e-3
    p = np.c_[rng.uniform(0, 11e-3, (n, 3)), np.full(n, 0.5 * d)]
    g = sg.build_graph(torch.from_numpy(p).to(DEV), sg.make_grid((0, 0, 0), (11e-3,) * 3, d))
    gen = torch.Generator(device=DEV).manual_seed(1)
    xn = (torch.randn((n, sg.NODE_IN), device=DEV, generator=gen) * 0.5).to(torch.bfloat16)
    target = torch.randn((n, 6), device=DEV, generator=gen)
    out = {}
    for path in (1, 0):
        assert lib.sdem_sg_set_tensor_path(path) == 0
        try:
            net = sg.Network(seed=2)
            net.lib = Calls(lib)
            y = net.forward(g, xn, keep=False)
            net.train_step(g, xn, target)
            assert ("sdem_sg_mlp" in net.lib.names) == (path == 1)
            out[path] = (y, net.grad.clone(), net.p.clone())
        finally:
            assert lib.sdem_sg_set_tensor_path(1) == 0
    for a, b in zip(out[0], out[1]):
        assert torch.equal(a, b)
