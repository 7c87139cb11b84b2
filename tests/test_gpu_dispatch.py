"""Which kernels a call takes at both sides of the lines that its rules draw (the results on either side are held against fp64 and against the separate calls
in test_gpu_mlp_chain.py and test_gpu_train_step.py)."""
import pytest

from graph_kernels import kernels

pytestmark = pytest.mark.gpu


def _network(lib, batch, I, dims):
    net = lib.Mlp(I, dims, ["relu"] * (len(dims) - 1) + ["identity"], batch)
    net.params.uniform_(-0.1, 0.1)
    return net


@pytest.mark.parametrize("batch,chunks,I,dims,one_launch", [
    (1024, 1, 64, [256, 256, 256, 16], True), (2048, 1, 64, [256, 256, 256, 16], False), (8192, 1, 64, [256, 256, 256, 16], False), (2048, 1, 64, [256, 256, 16], True),
    (4096, 1, 64, [256, 256, 16], False), (5003, 1, 33, [200, 200, 7], True), (8192, 1, 64, [64, 64, 64, 16], True), (8192, 1, 64, [128, 128, 128, 16], False), (8192, 1, 64, [100, 100, 100, 16], False),
    (1024, 4, 64, [128, 128, 128, 16], True), (512, 8, 64, [256, 256, 16], True),
    (4096, 2, 64, [256, 256, 256, 16], False), (2048, 1, 64, [320, 320, 16], True), (8192, 1, 64, [320, 320, 16], False)])
def test_training_step_takes_one_launch_where_that_is_faster(lib, batch, chunks, I, dims, one_launch):
    import torch
    net = _network(lib, batch, I, dims)
    x, y = torch.randn(batch * chunks, I, device="cuda"), torch.randn(batch * chunks, dims[-1], device="cuda")
    names = kernels(lambda: net.train_step(x, y, 1.0 / chunks))
    assert (len(names) == 1 and "mlp_team_step" in names[0]) == one_launch, names


@pytest.mark.parametrize("batch,I,dims,one_launch", [
    (3072, 64, [320, 320, 16], False), (3072, 512, [128, 128, 10], True), (6144, 64, [128, 128, 128, 16], True), (512, 128, [350, 350, 10], True), (1024, 128, [350, 350, 10], False),
    (256, 100, [256, 256, 256, 256], True), (512, 100, [256, 256, 256, 256], False), (128, 32, [512, 512, 4], False)])
def test_training_step_beside_kernels_per_layer_takes_one_launch_where_that_is_faster(lib, batch, I, dims, one_launch):
    test_training_step_takes_one_launch_where_that_is_faster(lib, batch, 1, I, dims, one_launch)


def _chain(names):
    return any("mlp_chain_kernel" in n for n in names)


@pytest.mark.parametrize("rows,I,dims,evaluate,forward,gradients,d_input", [
    (2048, 64, [256, 256, 256, 16], True, True, True, True), (2047, 64, [256, 256, 256, 16], False, False, False, False), (2048, 33, [200, 200, 7], True, False, True, True),
    (4096, 33, [200, 200, 7], True, True, True, True), (2048, 17, [130, 130, 3], True, False, False, False), (8192, 17, [130, 130, 3], True, True, True, True),
    (4096, 64, [256, 16], True, True, False, True), (8192, 8, [256, 4], False, False, False, True), (16384, 8, [256, 4], True, True, True, True), (16384, 64, [256], False, False, False, False),
    (8191, 27, [64, 64, 8], False, False, False, False), (8192, 27, [64, 64, 8], True, False, True, True), (16384, 27, [64, 64, 8], True, True, True, True),
    (8192, 64, [64, 4], False, False, False, True), (16384, 20, [32, 32, 32, 8], True, True, True, True), (65536, 4, [32, 32, 15], True, False, True, True),
    (65536, 64, [64, 4], True, False, True, True)])
def test_passes_of_a_network_take_the_chain_kernels_where_those_are_faster(lib, rows, I, dims, evaluate, forward, gradients, d_input):
    import torch
    net = _network(lib, rows, I, dims)
    x, d, g = torch.randn(rows, I, device="cuda"), torch.randn(rows, dims[-1], device="cuda"), torch.empty(rows, I, device="cuda")
    y = torch.empty(rows, dims[-1], device="cuda")
    got = [_chain(kernels(call)) for call in (lambda: net.evaluate(x, y), lambda: net.forward(x), lambda: net.backward(x, d),
                                              lambda: net.backward(x, d, d_input=g, accumulate_gradients=False))]
    assert got == [evaluate, forward, gradients, d_input]
