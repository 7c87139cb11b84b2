"""The grid-wide barrier of the cooperative launches: a wait that runs into its limit is reported, leaves the barrier clean for its next launch and stops
the calls that need one until it is cleared; captured launches share no barrier with the others."""
import ctypes as C

import pytest

import __graft_entry__ as entry

pytestmark = pytest.mark.gpu


class Barrier(C.Structure):
    _fields_ = [("words", C.c_void_p), ("status", C.c_void_p)]


@pytest.fixture(scope="module")
def case(lib):
    lib.lib()
    L = C.CDLL(entry.build_barrier_test())
    L.barrier_case_take.argtypes = [C.POINTER(Barrier), C.c_void_p]
    L.barrier_case_run.argtypes = [C.POINTER(Barrier), C.c_int, C.c_int, C.c_void_p, C.c_void_p]
    L.barrier_case_words.argtypes = [C.POINTER(Barrier), C.c_void_p]
    return L


def _status(lib):
    import torch
    torch.cuda.synchronize()
    pass_status, state = C.c_int(-1), C.c_int(-1)
    assert lib.lib().b200rl_cooperative_pass_status(C.byref(pass_status)) == 0
    assert lib.lib().b200rl_device_error_state(C.byref(state)) == 0
    return pass_status.value, state.value


def _network(lib, batch=256, extra=0):
    net = lib.Mlp(4, [64, 64, 1], ["relu", "relu", "identity"], batch, extra_params=extra)
    net.params.uniform_(-0.3, 0.3)
    return net


def _epoch(lib, actor, critic):
    import torch
    from rl_tools_b200 import ppo
    layout = ppo.DatasetLayout(4, 1)
    ppo.train(actor, critic, torch.rand(512, layout.data_dim, device="cuda"), layout, 512, 256, n_epochs=1)


def test_a_wait_that_runs_into_its_limit(lib, case):
    import torch
    assert _status(lib) == (0, 0)
    bar, words = Barrier(), (C.c_uint * 4)()
    stream = torch.cuda.current_stream().cuda_stream
    assert case.barrier_case_take(C.byref(bar), stream) == 0

    def run(absent):
        passed = torch.full((8,), -1, device="cuda", dtype=torch.int32)
        assert case.barrier_case_run(C.byref(bar), 8, absent, passed.data_ptr(), stream) == 0
        torch.cuda.synchronize()
        assert case.barrier_case_words(C.byref(bar), words) == 0
        return passed.tolist(), list(words)

    actor, critic = _network(lib, extra=1), _network(lib)
    x, y = torch.randn(256, 4, device="cuda"), torch.randn(256, 1, device="cuda")
    critic.train_step(x, y)
    try:
        assert run(0) == ([1] * 8, [0] * 4) and _status(lib) == (0, 0)
        assert run(2) == ([-1, -1] + [0] * 6, [0] * 4)          # six CTAs wait for two that never come: about a second
        assert _status(lib) == (1, 1)
        assert run(0) == ([1] * 8, [0] * 4)                     # the same barrier
        assert _status(lib) == (1, 1)
        for call in (lambda: critic.train_step(x, y), lambda: _epoch(lib, actor, critic)):
            with pytest.raises(lib.B200RLError, match="status 4"):
                call()
    finally:
        assert lib.lib().b200rl_device_error_clear() == 0
    assert _status(lib) == (0, 0)
    critic.train_step(x, y)
    _epoch(lib, actor, critic)
    assert _status(lib) == (0, 0)


@pytest.mark.parametrize("I,dims,batch", [(4, [256, 256, 1], 256), (4, [64, 64, 1], 1000), (33, [200, 200, 7], 5003)])
def test_the_kernels_that_wait_at_one_leave_no_status(lib, I, dims, batch):
    import torch
    net = lib.Mlp(I, dims, ["relu", "relu", "identity"], batch)
    net.params.uniform_(-0.1, 0.1)
    for _ in range(3):
        net.train_step(torch.randn(batch, I, device="cuda"), torch.randn(batch, dims[-1], device="cuda"))
    _epoch(lib, _network(lib, extra=1), _network(lib))
    assert _status(lib) == (0, 0)


def test_replays_beside_more_launches_than_there_are_barriers_to_hand_round(lib):
    """A graph keeps the barrier of its capture. Its replays run beside 20,000 launches on another stream, more than the ring that those take theirs from; both
    networks end up where they do alone."""
    import torch
    x, y = torch.randn(256, 4, device="cuda"), torch.randn(256, 1, device="cuda")
    side, results = torch.cuda.Stream(), []
    for together in (False, True):
        torch.manual_seed(1)
        a, b = _network(lib), _network(lib)
        a.train_step(x, y)
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=side):
            a.train_step(x, y)
        torch.cuda.synchronize()
        for k in range(20000):
            if k % 4 == 0:
                with torch.cuda.stream(side):
                    graph.replay()
                if not together:
                    torch.cuda.current_stream().wait_stream(side)
            b.train_step(x, y)
            if not together and k % 4 == 3:
                side.wait_stream(torch.cuda.current_stream())
        torch.cuda.synchronize()
        results.append([t.clone() for n in (a, b) for t in (n.params, n.m, n.v)])
        del graph
    assert _status(lib) == (0, 0)
    for alone, beside in zip(*results):
        assert torch.equal(alone, beside)
