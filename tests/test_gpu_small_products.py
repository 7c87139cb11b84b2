"""Kernels of small problems at the edges of their tiles: forward products (32 x 16 outputs, 256 summed indices), the backward launches of wide networks at
small batches (32 x 32 outputs, 256 summed indices), the advantage recurrence (1,024 steps at a time) and the row shuffle (64 rows at a time)."""
import numpy as np
import pytest

import make_golden as mg

pytestmark = pytest.mark.gpu


def matrix(torch, seed, rows, cols, pad=0):
    wide = torch.zeros(rows, cols + pad, device="cuda")
    wide[:, pad:] = torch.from_numpy(mg.det_normal(seed, rows * cols).reshape(rows, cols)).cuda()
    return wide[:, pad:]


@pytest.mark.parametrize("pad", [0, 1, 4])
@pytest.mark.parametrize("rows,I,O", [(1, 1, 1), (31, 255, 15), (32, 256, 16), (33, 257, 17), (256, 300, 2), (1000, 516, 100), (4600, 5, 33), (7, 1030, 260)])
def test_small_forward(lib, rows, I, O, pad):
    import torch
    net = lib.Mlp(I, [O], ["tanh"], rows)
    net.params.copy_(torch.from_numpy(mg.det_uniform(3, net.params.numel()) / np.float32(np.sqrt(I))).cuda())
    x = matrix(torch, 1, rows, I, pad)
    W, b = net.params[:O * I].view(O, I).double(), net.params[O * I:].double()
    want = x.double() @ W.T + b
    net.forward(x)
    assert float((net.pre.view(rows, O).double() - want).abs().max()) <= 2e-6
    assert float((net.output().double() - want.tanh()).abs().max()) <= 2e-6
    assert torch.equal(net.evaluate(x), net.output())


@pytest.mark.parametrize("batch,I,dims,acts", [(1, 3, [300, 1], ["relu", "identity"]), (256, 4, [256, 256, 1], ["relu", "relu", "identity"]), (257, 35, [257, 130, 3], ["tanh", "relu", "tanh"]),
                                               (512, 512, [300, 512, 64, 33], ["tanh", "sigmoid", "relu", "identity"]), (33, 130, [260], ["tanh"])])
@pytest.mark.parametrize("mode", ["gradients", "both", "input"])
def test_backward_of_wide_networks(lib, batch, I, dims, acts, mode):
    import torch
    act = {"identity": lambda v: v, "relu": torch.relu, "tanh": torch.tanh, "sigmoid": torch.sigmoid}
    net = lib.Mlp(I, dims, acts, batch)
    net.params.copy_(torch.from_numpy(mg.det_uniform(5, net.params.numel()) * np.float32(0.08)).cuda())
    x, d_out = matrix(torch, 1, batch, I), matrix(torch, 2, batch, dims[-1])
    params, xs = net.params.double().requires_grad_(), x.double().requires_grad_()
    h, off, fan_in = xs, 0, I
    for d, a in zip(dims, acts):
        h = act[a](h @ params[off:off + d * fan_in].view(d, fan_in).T + params[off + d * fan_in:off + d * fan_in + d])
        off += d * fan_in + d; fan_in = d
    (h * d_out.double()).sum().backward()
    net.grads.fill_(0.5)
    d_input = torch.zeros(batch, I, device="cuda") if mode != "gradients" else None
    net.forward(x)
    net.backward(x, d_out.clone(), d_input=d_input, accumulate_gradients=mode != "input")

    def close(got, want):
        assert float((got - want).abs().max()) <= 2e-5 * float(want.abs().max()) + 1e-6
    close(net.grads.double(), params.grad + 0.5 if mode != "input" else torch.full_like(params, 0.5))
    if d_input is not None:
        close(d_input.double(), xs.grad)


@pytest.mark.parametrize("n_envs,steps", [(1, 1), (3, 1023), (2, 1024), (5, 1025), (2, 3000), (300, 9)])
def test_advantages_over_chunks_of_steps(lib, n_envs, steps):
    import torch
    rows = n_envs * (steps + 1)
    rs = np.random.RandomState(steps)
    r, v = rs.randn(rows).astype(np.float32), rs.randn(rows).astype(np.float32)
    te = (rs.rand(rows) < 0.01).astype(np.float32)
    tr = np.maximum(te, (rs.rand(rows) < 0.01).astype(np.float32))
    column = lambda a: torch.from_numpy(a).cuda()
    adv, tgt = lib.gae(column(r), column(v), column(te), column(tr), n_envs, steps, 0.99, 0.95)
    want, f = np.zeros((steps, n_envs), np.float32), np.float32
    R, V, TE, TR = (a.reshape(steps + 1, n_envs) for a in (r, v, te, tr))
    lg = f(0.95) * f(0.99)
    previous = np.zeros(n_envs, f)
    for t in range(steps - 1, -1, -1):                          # the recurrence in the reference's order of operations, fp32 throughout
        td = (R[t] + f(0.99) * np.where(TE[t] != 0, f(0), V[t + 1])) - V[t]
        td = np.where((TR[t] != 0) & (TE[t] == 0), f(0), td)
        previous = lg * np.where(TR[t] != 0, f(0), previous) + td
        want[t] = previous
    assert np.array_equal(adv.cpu().numpy().reshape(steps, n_envs), want)
    assert np.array_equal(tgt.cpu().numpy().reshape(steps, n_envs), want + V[:steps])


@pytest.mark.parametrize("rows,cols,picked", [(1, 5, [0]), (63, 7, [0, 2, 6]), (64, 64, list(range(64))), (65, 70, [1, 5, 33, 63]), (1000, 12, [0, 1, 2, 7, 11])])
def test_permuted_columns(lib, rows, cols, picked):
    import torch
    data = matrix(torch, 4, rows, cols).contiguous()
    before, perm = data.clone(), torch.randperm(rows, device="cuda").int()
    lib.permute_rows(data, rows, perm, picked)
    want = before.clone()
    want[:, picked] = before[perm.long()][:, picked]
    assert torch.equal(data, want)
