"""What BasisNet.train refuses before anything is launched."""

import types

import pytest
import torch

from impuritymodel_gb300.pruning import BasisNet


class _Launched(Exception):
    pass


def _net(device):
    def launch(*args):
        raise _Launched

    net = object.__new__(BasisNet)
    lib = types.SimpleNamespace(edgpu_mlp_step_workspace=launch, edgpu_mlp_train_step=launch)
    net.eng = types.SimpleNamespace(device=torch.device(device), lib=lib, stream=None)
    return net


@pytest.mark.parametrize("states,log_w", [
    (torch.zeros((256, 5), dtype=torch.int64), torch.zeros(255)),             # a weight short
    (torch.zeros((256, 5), dtype=torch.int64), torch.zeros(0)),
    (torch.zeros((256, 5), dtype=torch.int32), torch.zeros(256)),             # half of each word
    (torch.zeros((256, 5), dtype=torch.int64, device="meta"), torch.zeros(256)),  # on another device
    (torch.zeros((256, 5), dtype=torch.int64), torch.zeros(256, device="meta")),
])
def test_train_refuses(states, log_w):
    with pytest.raises(ValueError):
        _net("cpu").train(states, log_w, epochs=1, batch=128)


@pytest.mark.parametrize("states,log_w", [
    (torch.zeros((256, 5), dtype=torch.int64), torch.zeros(256)),
    (torch.zeros((256, 2), dtype=torch.int64), torch.zeros(300)),  # more weights than states
    (torch.zeros((256, 5), dtype=torch.int64), torch.zeros(256, dtype=torch.float64)),
    (torch.zeros((256, 10), dtype=torch.int64)[:, ::2], torch.zeros(512)[::2]),
])
def test_train_takes(states, log_w):
    with pytest.raises(_Launched):
        _net("cpu").train(states, log_w, epochs=1, batch=128)
