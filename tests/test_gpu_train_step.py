"""The one-call training step (b200rl_mlp_train_step) and the one-call PPO epoch (b200rl_ppo_train_epoch) against the sequences of separate calls
they stand for, at the sizes where their kernels can go wrong: rows that fill no tile, one row, widths that are no multiple of four, every team
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


@pytest.mark.parametrize("batch,minibatches,obs,actions,hidden,act,options", [
    (512, 3, 3, 1, 64, "relu", {}), (2048, 2, 27, 8, 64, "tanh", {}), (97, 4, 5, 3, 32, "tanh", {}), (1000, 2, 18, 5, 100, "relu", dict(normalize_advantage=False)),
    (30, 70, 4, 2, 16, "tanh", dict(learn_action_std=False))])
def test_ppo_epoch_equals_the_separate_calls(lib, batch, minibatches, obs, actions, hidden, act, options):
    import torch
    from rl_tools_b200 import ppo
    layout = ppo.DatasetLayout(obs, actions)
    rows = batch * minibatches
    data = mg.det_normal(3, rows * layout.data_dim).reshape(rows, layout.data_dim).astype(np.float32)
    data[:, layout.action_log_probs] = data[:, layout.action_log_probs] * 0.5 - actions
    dataset = torch.from_numpy(data).cuda()
    acts = [act, act, "identity"]
    nets = [[_net(lib, torch, batch, obs, [hidden, hidden, actions], acts, 20, extra=actions), _net(lib, torch, batch, obs, [hidden, hidden, 1], acts, 30)] for _ in range(2)]
    for actor, _ in nets:
        actor.extra("params").fill_(-0.5)
    full = dict(epsilon_clip=0.2, entropy_coefficient=0.01, advantage_epsilon=1e-8, normalize_advantage=True, learn_action_std=True)
    full.update(options)
    assert ppo._train_epoch(*nets[0], dataset, layout, minibatches, batch, **full)
    for k in range(minibatches):
        ppo._minibatch_update(*nets[1], dataset[k * batch:(k + 1) * batch], layout, **full)
    for got, want in zip(*nets):
        for name in ("params", "v", "m", "grads"):
            _close(getattr(got, name), getattr(want, name), 2e-6 if name in ("params", "v") else 2e-4)
        assert torch.equal(got.adam_state, want.adam_state)


@pytest.mark.parametrize("batch,I,dims,acts", [
    (3, 1, [1], ["tanh"]), (33, 4, [4, 4], ["tanh", "identity"]), (300, 3, [5, 9, 2], ["tanh", "sigmoid", "identity"]), (1024, 16, [64, 64, 6], ["tanh", "tanh", "tanh"]),
    (2049, 31, [30, 66, 3], ["fast_tanh", "tanh", "identity"]), (64, 200, [130, 17, 8], ["tanh", "tanh", "identity"]), (1025, 12, [96, 100, 104, 1], ["tanh", "tanh", "sigmoid", "identity"]),
    (700, 64, [256, 256, 256, 5], ["tanh", "tanh", "tanh", "identity"]), (400, 511, [508, 12], ["tanh", "identity"]),
    (700, 64, [320, 320, 16], ["tanh", "tanh", "identity"]), (259, 13, [309, 311, 3], ["tanh", "tanh", "tanh"])])
def test_train_step_of_tiles_and_patches(lib, batch, I, dims, acts):
    """Sizes at which the walk's tiles have remainders: one unit, inputs that are and are not whole pieces of four (the bias lies in a piece of its own or in the last one), a summed index
    shared out over one to sixteen lanes, each size of gradient patch, odd numbers of patches, aligned and unaligned input rows."""
    test_train_step_equals_the_separate_calls(lib, batch, 1, I, dims, acts)
    test_train_step_equals_the_separate_calls(lib, batch, 2, I, dims, acts)


@pytest.mark.parametrize("batch,I,dims,acts", [
    (40, 5, [16, 6], ["tanh", "relu"]), (40, 5, [16, 6], ["tanh", "tanh"]), (40, 5, [16, 6], ["relu", "identity"]), (256, 4, [256, 256, 1], ["relu", "relu", "relu"]),
    (256, 4, [256, 255, 3], ["relu", "tanh", "fast_tanh"])])
@pytest.mark.parametrize("value", [float("nan"), float("inf")])
def test_train_step_keeps_what_is_not_finite(lib, batch, I, dims, acts, value):
    """A target that is not finite reaches the gradient also where the derivative of its output, or of the units below it, is 0 (inactive ReLU, saturated tanh): the same entries are finite
    and the same are NaN as after the separate calls."""
    import torch
    x = torch.from_numpy(mg.det_normal(1, batch * I).reshape(batch, I)).cuda()
    a, b = _net(lib, torch, batch, I, dims, acts, 5), _net(lib, torch, batch, I, dims, acts, 5)
    n_last = dims[-1] * dims[-2] + dims[-1]
    for net in (a, b):
        net.params[-dims[-1]:] = -40.0                                    # every output far on the side where its derivative is 0, if its activation has one
    y = torch.from_numpy(mg.det_normal(2, batch * dims[-1]).reshape(batch, dims[-1])).cuda()
    y[batch // 2, dims[-1] // 2] = value
    a.train_step(x, y, 1.0)
    b.zero_gradient()
    out = b.forward(x)
    b.backward(x, lib.mse_gradient(out, y, 1.0, d_a=b.d_out_buffer()))
    b.step()
    assert not torch.isfinite(b.grads[-n_last:]).all()
    for name in ("grads", "params", "m", "v"):
        got, want = getattr(a, name), getattr(b, name)
        assert torch.equal(torch.isfinite(got), torch.isfinite(want)), name
        if value != value:
            assert torch.equal(torch.isnan(got), torch.isnan(want)), name


@pytest.mark.parametrize("rows,I,dims", [(256, 4, [256, 256, 1]), (5003, 33, [200, 200, 7]), (1024, 64, [64, 64, 64, 16]), (337, 8, [256, 256, 256, 3])])
def test_the_plan_of_a_step_costs_little(lib, rows, I, dims):
    """Every one-launch step looks for its plan among 32 candidates; the size query does nothing else of weight. 0.7 to 0.9 us, 4.9 to 7.2 where everything the kernel needs was made for each
    of the candidates (least of many calls, less those of a call that returns at once)."""
    import ctypes
    import time
    shape = lib.MlpShape.make(I, dims, ["tanh"] * len(dims))
    query = lib.lib().b200rl_mlp_backward_scratch_bytes

    def least(batch):
        best = 1.0
        for _ in range(100):
            begin = time.perf_counter()
            for _ in range(50):
                query(ctypes.byref(shape), batch)
            best = min(best, (time.perf_counter() - begin) / 50)
        return best
    assert least(rows) - least(0) < 3e-6                                  # between the two, with room for a slower host


@pytest.mark.parametrize("batch,I,dims", [(256, 4, [256, 256, 1]), (2048, 64, [64, 64, 16]), (700, 64, [320, 320, 16])])
def test_every_cta_steps_with_the_age_of_its_step(lib, batch, I, dims):
    """The first steps of an optimizer, whose corrections differ most from one to the next: each equals the optimizer's own kernel on the same gradients, in every parameter."""
    import torch
    acts = ["tanh"] * (len(dims) - 1) + ["identity"]
    net, other = _net(lib, torch, batch, I, dims, acts, 5), _net(lib, torch, batch, I, dims, acts, 5)
    for n in (net, other):
        n.m.zero_(); n.v.zero_()
        n.adam_state[0] = 1
    x = torch.from_numpy(mg.det_normal(1, batch * I).reshape(batch, I)).cuda()
    y = torch.from_numpy(mg.det_normal(2, batch * dims[-1]).reshape(batch, dims[-1])).cuda()
    for step in range(100):
        net.train_step(x, y, 1.0)
        other.grads.copy_(net.grads)
        other.step()
        for name in ("params", "m", "v", "adam_state"):
            assert torch.equal(getattr(net, name), getattr(other, name)), (step, name)


@pytest.mark.parametrize("batch,I,dims,ctas", [
    (838, 12, [16, 16, 3], (20, 60)), (508, 5, [16, 16, 14], (20, 60)), (500, 3, [32, 32, 1], (25, 64)),       # a tile of several rows per CTA: fewer CTAs at the barrier
    (50, 5, [100, 100, 2], (26, 104)), (80, 24, [100, 100, 2], (40, 148)), (700, 5, [100, 100, 100, 2], (100, 148)),      # few rows of wider layers: teams of several CTAs
    (300, 20, [64, 64, 3], (60, 90))])
def test_small_steps_are_spread_over_as_many_ctas_as_pay(lib, tmp_path, batch, I, dims, ctas):
    """The plan's CTAs, whose number the launch shows; and the step by that plan against the separate calls."""
    import json
    import torch
    from torch.profiler import ProfilerActivity, profile
    net = _net(lib, torch, batch, I, dims, ["tanh"] * len(dims), 5)
    x, y = torch.zeros(batch, I, device="cuda"), torch.zeros(batch, dims[-1], device="cuda")
    net.train_step(x, y, 1.0)
    torch.cuda.synchronize()
    with profile(activities=[ProfilerActivity.CUDA]) as prof:
        net.train_step(x, y, 1.0)
        torch.cuda.synchronize()
    prof.export_chrome_trace(str(tmp_path / "trace.json"))
    with open(tmp_path / "trace.json") as f:
        grids = [e["args"]["grid"] for e in json.load(f)["traceEvents"] if e.get("cat") == "kernel" and "mlp_team_step" in e["name"]]
    assert len(grids) == 1 and ctas[0] <= grids[0][0] <= ctas[1], grids
    test_train_step_equals_the_separate_calls(lib, batch, 1, I, dims, ["tanh"] * (len(dims) - 1) + ["identity"])
