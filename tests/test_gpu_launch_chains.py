"""Kernels that are launched before the one in front of them has ended (they wait for it on the device): a chain of dependent calls gives the bits of the same calls made one by one, with the
device idle in between; on a stream, and captured as a graph with a second branch."""
import pytest

pytestmark = pytest.mark.gpu


def _chain(lib, torch, hidden, batch, meet, branch):
    """Ten updates of a network and of its copy's target, every call reading what the call before has written; meet() after each of them."""
    dims, acts = [hidden, hidden, 2], ["relu", "tanh", "identity"]
    gen = torch.Generator(device="cuda"); gen.manual_seed(hidden + batch)
    net, target = lib.Mlp(5, dims, acts, batch), lib.Mlp(5, dims, acts, batch)
    net.params.copy_((torch.rand(net.params.shape, device="cuda", generator=gen) - 0.5) * 0.2)
    target.params.copy_(net.params)
    x, noise = torch.randn(batch, 5, device="cuda", generator=gen), torch.zeros(batch, 2, device="cuda")
    counter = torch.zeros(1, dtype=torch.int64, device="cuda")
    y, q = torch.empty(batch, 2, device="cuda"), torch.empty(batch, 2, device="cuda")
    side = torch.cuda.Stream()

    def update():
        lib.randn_device_rng(noise, 7, 1, call_counter=counter); meet()
        with branch(side):
            target.evaluate(x, y=q); meet()
        net.zero_gradient(); meet()
        out = net.forward(x); meet()
        branch.join(side)
        y.copy_(q); meet()
        lib.polyak_update(noise.view(1, -1), y.view(1, -1), 0.9); meet()
        net.backward(x, lib.mse_gradient(out, y, 1.0, d_a=net.d_out_buffer())); meet()
        net.step(); meet()
        lib.polyak_update(net.params.view(1, -1), target.params.view(1, -1), 0.99); meet()
        lib.counter_advance(counter, 1); meet()
    return update, [net.params, net.grads, net.m, net.v, net.adam_state, net.out, target.params, noise, y, q, counter]


class _Branch:
    def __init__(self, torch):
        self.torch = torch

    def __call__(self, stream):
        stream.wait_stream(self.torch.cuda.current_stream())
        return self.torch.cuda.stream(stream)

    def join(self, stream):
        self.torch.cuda.current_stream().wait_stream(stream)


@pytest.mark.parametrize("hidden,batch", [(256, 256), (256, 37), (64, 100), (32, 512), (130, 300)])
def test_a_chain_of_launches_has_the_bits_of_launches_one_by_one(lib, hidden, batch):
    import torch
    results = []
    for how in ("one by one", "stream", "graph"):
        update, state = _chain(lib, torch, hidden, batch, torch.cuda.synchronize if how == "one by one" else lambda: None, _Branch(torch))
        if how == "graph":
            start = [t.clone() for t in state]
            stream = torch.cuda.Stream()
            stream.wait_stream(torch.cuda.current_stream())
            with torch.cuda.stream(stream):
                update()
            torch.cuda.synchronize()
            graph = torch.cuda.CUDAGraph()
            with torch.cuda.graph(graph, stream=stream):
                update()
            for t, s in zip(state, start):
                t.copy_(s)
        for _ in range(10):
            graph.replay() if how == "graph" else update()
        torch.cuda.synchronize()
        results.append([t.clone() for t in state])
    for got in results[1:]:
        for a, b in zip(got, results[0]):
            assert torch.equal(a, b)


def _digest(torch, tensors):
    import hashlib
    h = hashlib.sha256()
    for t in tensors:
        h.update(t.detach().contiguous().cpu().numpy().tobytes())
    return h.hexdigest()


def _off_policy(pkg, loops, torch, quadrotor, hidden):
    """Runner step, replay sampling and SAC update, launch by launch: the environments' kernels, gather_batch, the sampling head, the target values and the min-value gradient."""
    import numpy as np
    import os
    torch.manual_seed(hidden)
    common = dict(hidden_dim=hidden, replay_capacity=1000, seed=hidden, use_graph=False)
    if quadrotor:
        fix = np.load(os.path.join(os.path.dirname(os.path.abspath(__file__)), "golden", "l2f.npz"))
        loop = loops.L2fSacLoop(pkg.L2fParameters.make(fix["dynamics"], float(fix["dt"])), fix["mdp"], fix["init"], n_envs=16, batch_size=100, **common)
    else:
        loop = loops.PendulumSacLoop(n_envs=3, batch_size=100, n_warmup_steps=50, episode_step_limit=40, **common)
    for _ in range(130):
        loop.step()
    a = loop.agent
    return [t for n in [a.actor] + a.critics for t in (n.params, n.grads, n.m, n.v)] + [t.params for t in a.critics_target] + [a.log_alpha, loop.states, loop.replay, loop.batch["oa_base"]]


def _many_rows(pkg, torch, I, dims, rows):
    """A training step over two chunks by the tensor-core kernels: padded inputs, chains, gradients, the reduction of their parts."""
    gen = torch.Generator(device="cuda"); gen.manual_seed(rows)
    net = pkg.Mlp(I, dims, ["tanh"] * (len(dims) - 1) + ["identity"], rows)
    net.params.copy_((torch.rand(net.params.shape, device="cuda", generator=gen) - 0.5) * 0.2)
    x, y = torch.randn(2 * rows, I, device="cuda", generator=gen), torch.randn(2 * rows, dims[-1], device="cuda", generator=gen)
    for _ in range(5):
        net.train_step(x, y, 0.5)
    return [net.params, net.grads, net.m, net.v, net.pre, net.out]


def _on_policy(loops, torch, n_envs, batch):
    """Collect, advantages, shuffled epochs as one call each: row permutation, the statistics of the advantages, the epoch kernel."""
    torch.manual_seed(batch)
    loop = loops.PendulumPpoLoop(n_envs=n_envs, steps_per_env=64, batch_size=batch, n_epochs=5, seed=3)
    for _ in range(3):
        loop.step()
    return [t for n in (loop.actor, loop.critic) for t in (n.params, n.grads, n.m, n.v)] + [loop.dataset]


def _all_digests():
    import importlib
    import json
    import torch
    import __graft_entry__ as entry
    pkg = entry.load_package()
    loops = importlib.import_module("rl_tools_b200.loops")
    out = {"pendulum 64": _off_policy(pkg, loops, torch, False, 64), "pendulum 256": _off_policy(pkg, loops, torch, False, 256), "quadrotor": _off_policy(pkg, loops, torch, True, 64),
           "29-64-64-5": _many_rows(pkg, torch, 29, [64, 64, 5], 16387), "33-200-200-7": _many_rows(pkg, torch, 33, [200, 200, 7], 16390), "ppo": _on_policy(loops, torch, 64, 512)}
    torch.cuda.synchronize()
    print(json.dumps({k: _digest(torch, v) for k, v in out.items()}))


def test_loops_and_large_steps_have_the_bits_of_launches_one_by_one():
    """The chains inside native calls: the same program with every launch waited for by the driver (CUDA_LAUNCH_BLOCKING) and without, the second twice."""
    import json
    import os
    import subprocess
    import sys
    here = os.path.dirname(os.path.abspath(__file__))

    def run(blocking):
        env = dict(os.environ, CUDA_LAUNCH_BLOCKING="1" if blocking else "0", PYTHONPATH=os.pathsep.join([os.path.dirname(here), here, os.path.join(here, "golden")]))
        r = subprocess.run([sys.executable, "-c", "import test_gpu_launch_chains as t; t._all_digests()"], env=env, capture_output=True, text=True, timeout=300)
        assert r.returncode == 0, r.stderr[-2000:]
        return json.loads(r.stdout.splitlines()[-1])

    want = run(True)
    assert len(want) == 6
    for _ in range(2):
        assert run(False) == want
