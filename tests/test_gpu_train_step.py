"""The one-call training step (b200rl_mlp_train_step) against the sequence of separate calls it stands for, at the sizes where their kernels can go wrong: rows that fill no tile, one row, widths that are no multiple of four, every team
size, several chunks, parameters outside the layers."""
import numpy as np
import pytest

import make_golden as mg

pytestmark = pytest.mark.gpu

NETS = [  # (batch, chunks, input, dims, activations); smooth activations for the large ones (a ReLU flips where a pre-activation rounds across 0)
    (1, 1, 9, [33, 5], ["relu", "identity"]), (50, 2, 3, [7], ["identity"]), (256, 1, 4, [256, 256, 1], ["tanh", "tanh", "identity"]),
    (129, 1, 20, [512, 300, 10], ["sigmoid", "tanh", "identity"]), (77, 3, 13, [100, 101, 5], ["tanh", "sigmoid", "tanh"]), (1000, 1, 33, [64, 64, 8], ["fast_tanh", "tanh", "identity"]),
    (337, 1, 8, [256, 256, 256, 3], ["tanh", "fast_tanh", "tanh", "identity"]), (8192, 1, 17, [64, 64, 1], ["tanh", "tanh", "identity"]), (4100, 2, 5, [128, 128, 2], ["relu", "tanh", "identity"]),
    (60, 1, 6, [16, 16, 16, 16, 2], ["relu", "relu", "relu", "relu", "identity"]),                # five layers: the sequence itself
]


def _net(lib, torch, batch, I, dims, acts, seed, extra=0):
    net = lib.Mlp(I, dims, acts, batch, extra_params=extra)
    off, fan_in = 0, I
    for l, d in enumerate(dims):
        n = d * fan_in + d
        net.params[off:off + n] = torch.from_numpy(mg.det_uniform(seed + l, n) / np.float32(np.sqrt(fan_in))).cuda()
        off += n; fan_in = d
    n = net.params.numel()
    net.m.copy_(torch.from_numpy(mg.det_normal(seed + 50, n) * np.float32(1e-3)))
    net.v.copy_(torch.from_numpy(np.abs(mg.det_normal(seed + 51, n)) * np.float32(1e-4) + np.float32(1e-5)))
    net.adam_state[0] = 40
    return net


def _close(got, want, tol=2e-6):
    assert torch_norm(got - want) <= tol * torch_norm(want) + 1e-12


def torch_norm(t):
    return float(t.double().norm())


@pytest.mark.parametrize("batch,chunks,I,dims,acts", NETS)
def test_train_step_equals_the_separate_calls(lib, batch, chunks, I, dims, acts):
    import torch
    rows = batch * chunks
    x = torch.from_numpy(mg.det_normal(1, rows * I).reshape(rows, I)).cuda()
    y = torch.from_numpy(mg.det_normal(2, rows * dims[-1]).reshape(rows, dims[-1])).cuda()
    a, b = _net(lib, torch, batch, I, dims, acts, 5, extra=2), _net(lib, torch, batch, I, dims, acts, 5, extra=2)
    for step in range(2):
        a.train_step(x, y, 1.0 / chunks, optimize=step == 0)
        b.zero_gradient()
        for c in range(0, rows, batch):
            out = b.forward(x[c:c + batch])
            b.backward(x[c:c + batch], lib.mse_gradient(out, y[c:c + batch], 1.0 / chunks, d_a=b.d_out_buffer()))
        if step == 0:
            b.step()
        for name in ("grads", "params", "m", "v", "pre", "out"):
            _close(getattr(a, name), getattr(b, name))
        assert int(a.adam_state[0]) == int(b.adam_state[0]) == 41
