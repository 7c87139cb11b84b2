"""All layers of a forward pass in one tensor-core kernel against fp64: the least rows it serves, rows that fill no tile of 128, more row tiles than
SMs, widths on both sides of the 64-column pieces and of the 128-column stacking, one and eight layers, strided and unaligned operands."""
import numpy as np
import pytest

import make_golden as mg

pytestmark = pytest.mark.gpu

NETS = [  # (rows, input, dims, activations)
    (2048, 64, [256, 256, 16], ["relu", "tanh", "identity"]), (2049, 130, [256, 130, 129, 16], ["sigmoid", "tanh", "fast_tanh", "identity"]), (5003, 33, [200, 200, 7], ["tanh", "tanh", "identity"]),
    (2200, 200, [33], ["tanh"]), (8192, 3, [64, 64, 2], ["fast_tanh", "tanh", "identity"]), (8193, 5, [16, 32, 48, 64, 80, 96, 112, 128], ["tanh"] * 8),
    (148 * 128 * 2 + 77, 17, [100, 65, 1], ["relu", "sigmoid", "tanh"]), (148 * 128 + 1, 256, [256, 144], ["identity", "relu"]),
]
ACT = {"identity": lambda v: v, "relu": lambda v: v.clamp(min=0), "tanh": lambda v: v.tanh(), "sigmoid": lambda v: v.sigmoid(),
       "fast_tanh": lambda v: (lambda c: c * (27 + c * c) / (27 + 9 * c * c))(v.clamp(-3, 3))}


@pytest.mark.parametrize("strided", [False, True])
@pytest.mark.parametrize("rows,I,dims,acts", NETS)
def test_forward_and_evaluate_match_fp64(lib, rows, I, dims, acts, strided):
    import torch
    net = lib.Mlp(I, dims, acts, rows)
    off, fan_in = 0, I
    for l, d in enumerate(dims):
        n = d * fan_in + d
        net.params[off:off + n] = torch.from_numpy(mg.det_uniform(7 + l, n) / np.float32(np.sqrt(fan_in))).cuda()
        off += n; fan_in = d
    x = torch.from_numpy(mg.det_normal(1, rows * I).reshape(rows, I)).cuda()
    x[:, 0] *= 1e-3                                             # columns of different magnitude, a row of zeros, a row of large values
    x[1] = 0; x[2] *= 1e4
    if strided:
        wide = torch.zeros(rows, I + 3, device="cuda")
        wide[:, 1:I + 1] = x
        x = wide[:, 1:I + 1]
    h, off, fan_in, pres, outs = x.double(), 0, I, [], []
    for d, a in zip(dims, acts):
        W, b = net.params[off:off + d * fan_in].double().view(d, fan_in), net.params[off + d * fan_in:off + d * fan_in + d].double()
        off += d * fan_in + d; fan_in = d
        pres.append(h @ W.T + b); h = ACT[a](pres[-1]); outs.append(h)
    y = net.evaluate(x)
    net.forward(x)
    state = np.zeros(1, np.int32)
    assert lib.lib().b200rl_device_error_state(state.ctypes.data) == 0 and state[0] == 0

    def close(got, want):                                       # row by row: a row's error follows the row's own magnitude
        err, size = (got.double() - want).norm(dim=1), want.norm(dim=1)
        assert float((err - 3e-6 * size).max()) <= 1e-6

    off = 0
    for d, p, o in zip(dims, pres, outs):
        close(net.pre[off:off + rows * d].view(rows, d), p); close(net.out[off:off + rows * d].view(rows, d), o)
        off += rows * d
    close(y, outs[-1])
