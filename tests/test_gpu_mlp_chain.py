"""All layers of a forward pass in one tensor-core kernel against fp64, and the passes that take the kernels per layer beside it (test_gpu_dispatch.py says which):
the least rows it serves, rows that fill no tile of 128, more row tiles than SMs, widths on both sides of the 64-column pieces and of the 128-column
stacking, one to eight layers, strided and unaligned operands."""
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


DERIVATIVE = {"identity": lambda v: v * 0 + 1, "relu": lambda v: (v > 0).to(v.dtype), "tanh": lambda v: 1 - v.tanh() ** 2, "sigmoid": lambda v: v.sigmoid() * (1 - v.sigmoid()),
              "fast_tanh": lambda v: 1 - ACT["fast_tanh"](v) ** 2}


@pytest.mark.parametrize("mode", ["gradients", "both", "input"])
@pytest.mark.parametrize("rows,I,dims,acts", [n for n in NETS if len(n[2]) > 1] + [((1 << 18) + 131, 12, [40, 24, 4], ["relu", "tanh", "tanh"]), (9000, 140, [136, 3], ["relu", "identity"])])
def test_backward_matches_fp64(lib, rows, I, dims, acts, mode):
    """Backward in the same kernels: more than one chunk of 2^18 rows, both operands on either side of 128 and 256 columns, unaligned widths; gradients are
    added to what is there, the input gradient alone leaves them untouched."""
    import torch
    net = lib.Mlp(I, dims, acts, rows)
    off, fan_in = 0, I
    for l, d in enumerate(dims):
        n = d * fan_in + d
        net.params[off:off + n] = torch.from_numpy(mg.det_uniform(7 + l, n) / np.float32(np.sqrt(fan_in))).cuda()
        off += n; fan_in = d
    x = torch.from_numpy(mg.det_normal(1, rows * I).reshape(rows, I)).cuda()
    x[:, 0] *= 1e-3                                             # a column of small values, a row of zeros, a row of large values
    x[1] = 0; x[2] *= 1e2
    d_out = torch.from_numpy(mg.det_normal(2, rows * dims[-1]).reshape(rows, dims[-1])).cuda() / rows
    d_out[:, 0] *= 1e-4
    net.forward(x)
    net.grads.copy_(torch.from_numpy(mg.det_normal(3, net.grads.numel())).cuda() * 1e-3)
    before = net.grads.clone()
    d_input = torch.zeros(rows, I, device="cuda") if mode != "gradients" else None
    d, widths = d_out.double(), [I] + list(dims)
    wants = [None] * len(dims)
    poff = np.cumsum([0] + [o * i + o for i, o in zip(widths, dims)])
    aoff = np.cumsum([0] + [rows * o for o in dims])
    for l in range(len(dims) - 1, -1, -1):
        i, o = widths[l], dims[l]
        pre = net.pre[aoff[l]:aoff[l] + rows * o].view(rows, o).double()
        inp = x.double() if l == 0 else net.out[aoff[l - 1]:aoff[l - 1] + rows * i].view(rows, i).double()
        d = d * DERIVATIVE[acts[l]](pre)
        wants[l] = (d.T @ inp, d.abs().T @ inp.abs(), d.sum(0), d.abs().sum(0))
        d = d @ net.params[poff[l]:poff[l] + o * i].double().view(o, i)
    net.backward(x, d_out.clone(), d_input=d_input, accumulate_gradients=mode != "input")
    state = np.zeros(1, np.int32)
    assert lib.lib().b200rl_device_error_state(state.ctypes.data) == 0 and state[0] == 0
    if mode == "input":
        assert torch.equal(net.grads, before)
    else:
        for l, (dW, size_W, db, size_b) in enumerate(wants):
            i, o = widths[l], dims[l]
            got = net.grads[poff[l]:poff[l + 1]].double() - before[poff[l]:poff[l + 1]].double()
            # the sum of the terms' magnitudes, and the rounding of the sum with what was there
            assert float(((got[:o * i].view(o, i) - dW).abs() - 2e-6 * size_W).max()) <= 1e-9, l
            assert float(((got[o * i:] - db).abs() - 2e-6 * size_b).max()) <= 1e-9, l
    if d_input is not None:
        err, size = (d_input.double() - d).norm(dim=1), d.norm(dim=1)
        assert float((err - 1e-5 * size).max()) <= 1e-6 / rows


@pytest.mark.parametrize("rows", [2048, 2051, 2080, 2367, 2368, 2369])
def test_gradients_of_fewer_units_than_ranges(lib, rows):
    """Two layers, each of whose gradients is one job: 74 ranges of the rows for the 148 SMs, more than the batch has units of 32 rows. A range without a unit leaves zeros."""
    test_backward_matches_fp64(lib, rows, 128, [256, 16], ["tanh", "identity"], "gradients")


@pytest.mark.parametrize("rows,I,dims,acts", [
    (16385, 64, [64, 64, 64], ["tanh", "relu", "identity"]), (16400, 1, [16, 32, 17, 33, 48, 64, 64, 1], ["tanh"] * 8), (2 * 2 * 148 * 128 + 5, 33, [32, 31, 64, 2], ["sigmoid", "tanh", "fast_tanh", "tanh"]),
    (16385, 65, [64, 64, 3], ["tanh", "tanh", "identity"]), (16385, 64, [64, 65, 3], ["tanh", "tanh", "identity"])])
def test_networks_of_at_most_64_columns(lib, rows, I, dims, acts):
    """The kernels of two CTAs per SM: both sides of their line, operands of one and of both halves of a piece, more row tiles than two per SM; with the tolerances of the tests above."""
    test_forward_and_evaluate_match_fp64(lib, rows, I, dims, acts, False)
    test_backward_matches_fp64(lib, rows, I, dims, acts, "both")


@pytest.mark.parametrize("rows,I,dims", [(2048, 64, [256, 256, 16]), (4099, 64, [256, 256, 16]), (2100, 200, [130, 129]), (8192, 27, [64, 64, 8]), (16390, 27, [64, 64, 8]), (8200, 100, [33, 128, 7])])
def test_weights_far_below_the_largest_of_their_layer(lib, rows, I, dims):
    """Every third output of a layer has weights 2^-24 of the layer's largest, and so has every third input (a column, which is an output of the
    backward chain): each output column, input-gradient column and gradient row is as close to fp64 as its own size asks for. Two fp16 parts hold 22 bits
    of an operand, so a product is off by 2^-21, and the truncating accumulation of a 64-column piece adds about as much: 1e-6 in all, for each product of a chain."""
    import torch
    net = lib.Mlp(I, dims, ["identity"] * len(dims), rows)
    off, fan_in, weights, biases = 0, I, [], []
    for l, d in enumerate(dims):
        W = torch.from_numpy(mg.det_uniform(7 + l, d * fan_in).reshape(d, fan_in) / np.float32(np.sqrt(fan_in))).cuda()
        W[::3] *= 2.0 ** -24
        W[:, 1::3] *= 2.0 ** -24
        net.params[off:off + d * fan_in] = W.flatten()
        bias = torch.from_numpy(mg.det_uniform(17 + l, d)).cuda()
        bias[::3] *= 2.0 ** -24
        net.params[off + d * fan_in:off + d * fan_in + d] = bias
        biases.append(bias.double())
        weights.append(W.double())
        off += d * fan_in + d; fan_in = d
    x = torch.from_numpy(mg.det_normal(1, rows * I).reshape(rows, I)).cuda()

    def close(got, want, products=1):
        err, size = (got.double() - want).norm(dim=0), want.norm(dim=0)
        assert float((err / size).max()) <= 1e-6 * products

    y = net.evaluate(x)
    net.forward(x)
    inp, off = x.double(), 0
    for W, b in zip(weights, biases):
        got = net.out[off:off + rows * len(W)].view(rows, len(W))
        off += rows * len(W)
        close(got, inp @ W.T + b)
        inp = got.double()
    close(y, inp)
    d_out = torch.from_numpy(mg.det_normal(2, rows * dims[-1]).reshape(rows, dims[-1])).cuda() / rows
    d_input = torch.zeros(rows, I, device="cuda")
    net.zero_gradient()
    net.backward(x, d_out.clone(), d_input=d_input)
    d, poff = d_out.double(), net.n_mlp
    for l in range(len(dims) - 1, -1, -1):
        o, i = weights[l].shape
        poff -= o * i + o
        if l == 0:
            size = d.abs().T @ x.double().abs()                 # the sum over the rows cancels: its terms' magnitudes
            assert float(((net.grads[poff:poff + o * i].view(o, i).double() - d.T @ x.double()).abs() / size).max()) <= 2e-6
        d = d @ weights[l]
    close(d_input, d, products=len(dims))


def test_a_network_that_only_evaluates_holds_no_backward_scratch(lib):
    """64-256-256-256-16 at 2^18 rows: 0.8 GB that only the backward pass uses."""
    import torch
    rows, dims = 1 << 18, [256, 256, 256, 16]
    before = torch.cuda.memory_allocated()
    net = lib.Mlp(64, dims, ["relu"] * 3 + ["identity"], rows)
    x = torch.zeros(rows, 64, device="cuda")
    net.evaluate(x)
    net.forward(x)
    arenas = sum(t.numel() * t.element_size() for t in (net.params, net.grads, net.m, net.v, net.tick, net.tock, net.pre, net.out, net.workspace, x))
    assert net.scratch_bytes > 1 << 29 and torch.cuda.memory_allocated() - before < arenas + (1 << 26)
    net.backward(x, torch.zeros(rows, 16, device="cuda"))
    assert net.scratch.numel() == net.scratch_bytes


def test_gradients_of_many_rows(lib):
    """2^18 rows in one chunk: a bias gradient sums 12,500 of them per CTA. In sums of 256 values and sums of those it loses what the d_pre themselves lack, 3e-7
    in all; 6e-7 leaves room for other seeds (one running sum: 1.2e-6). A weight gradient adds 390 units of 32 rows per CTA; in four sums of a hundred it loses 2.5e-7
    where d_pre is nearly exact, in the last two layers (in one: 3.8e-7)."""
    import torch
    rows, I, dims, acts = 1 << 18, 64, [256, 256, 256, 16], ["tanh", "tanh", "tanh", "identity"]
    net = lib.Mlp(I, dims, acts, rows)
    gen = torch.Generator(device="cuda"); gen.manual_seed(3)
    off, fan_in = 0, I
    for d in dims:
        n = d * fan_in + d
        net.params[off:off + n] = (torch.rand(n, device="cuda", generator=gen) * 2 - 1) / fan_in ** 0.5
        off += n; fan_in = d
    x, d_out = torch.randn(rows, I, device="cuda", generator=gen), torch.randn(rows, dims[-1], device="cuda", generator=gen) / rows
    net.forward(x)
    net.zero_gradient()
    net.backward(x, d_out.clone())
    d, poff, aoff = d_out.double(), net.n_mlp, net.pre.numel()
    for l in range(len(dims) - 1, -1, -1):
        o, i = dims[l], dims[l - 1] if l else I
        poff -= o * i + o; aoff -= rows * o
        d = d * DERIVATIVE[acts[l]](net.pre[aoff:aoff + rows * o].view(rows, o).double())
        want = d.sum(0)
        assert float((net.grads[poff + o * i:poff + o * i + o].double() - want).norm() / want.norm()) <= 6e-7
        want = d.T @ (net.out[aoff - rows * i:aoff].view(rows, i) if l else x).double()
        assert float((net.grads[poff:poff + o * i].view(o, i).double() - want).norm() / want.norm()) <= (3.1e-7 if l >= 2 else 6e-7)
        d = d @ net.params[poff:poff + o * i].double().view(o, i)
