"""Folding a batch norm into a convolution's bias (host): parameters on different devices never reach the
kernel, which reads all of them on one."""

import pytest
import torch

import fvdb.nn as fvnn
from fvdb.nn import modules


def test_a_bias_on_another_device_is_left_to_torch(monkeypatch):
    conv = fvnn.SparseConv3d(4, 6, 3)
    conv.bias = torch.nn.Parameter(conv.bias.detach().to("meta"))
    monkeypatch.setattr(modules, "plain_cuda", lambda *t: True)  # two devices, as two GPUs would be

    class NoKernel:
        def __getattr__(self, name):
            raise AssertionError(f"{name} must not be called")

    monkeypatch.setattr(modules._lib, "load", lambda: NoKernel())
    with pytest.raises(RuntimeError):
        conv._folded((torch.ones(6), torch.zeros(6)))
