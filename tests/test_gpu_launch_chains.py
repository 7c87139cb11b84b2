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
