"""Host-side mirror of the reference's PPO update on the on-policy dataset matrix, driving the C ABI.

`DatasetLayout` gives the column views of rl/components/on_policy_runner/on_policy_runner.h:38-72 (symmetric observations);
`estimate_generalized_advantages` and `train` follow rl/algorithms/ppo/operations_generic.h:59-95 and :96-336 with the default
parameters of rl/algorithms/ppo/ppo.h:13-38. Everything runs on the GPU on torch CUDA tensors; there is no CPU path.
"""
import ctypes as C

from . import lib, check, _ptr, _stream, gae as _gae, mse_gradient as _mse_gradient, ppo_policy_gradient as _ppo_policy_gradient, permute_rows_scratch as _permute_rows_scratch


class DatasetLayout:
    """Column offsets of the dataset matrix [(steps + 1) * n_envs, data_dim], row = step * n_envs + env."""

    def __init__(self, observation_dim, action_dim):
        o, a = observation_dim, action_dim
        self.observation_dim, self.action_dim = o, a
        self.observations = slice(0, o)
        self.actions_mean = slice(o, o + a)
        self.actions = slice(o + a, o + 2 * a)
        self.action_log_probs = o + 2 * a
        self.rewards = o + 2 * a + 1
        self.terminated = o + 2 * a + 2
        self.truncated = o + 2 * a + 3
        self.reset = o + 2 * a + 4
        self.values = o + 2 * a + 5
        self.advantages = o + 2 * a + 6
        self.target_values = o + 2 * a + 7
        self.data_dim = o + 2 * a + 8


def estimate_generalized_advantages(dataset, layout, n_envs, steps, gamma=0.99, lam=0.95, ignore_termination=False):
    """Fills the advantage and target-value columns from rewards / values / flags, in place (one backward scan per environment).
    The value column must hold the critic's values of all (steps + 1) * n_envs observations."""
    rows = steps * n_envs
    _gae(dataset[:, layout.rewards], dataset[:, layout.values], dataset[:, layout.terminated], dataset[:, layout.truncated],
         n_envs, steps, gamma, lam, ignore_termination, advantages=dataset[:rows, layout.advantages], target_values=dataset[:rows, layout.target_values])
    return dataset


def _values_work(critic, n):
    """Work buffers of evaluate_values for n rows, kept with the critic."""
    import torch
    # As many rows per call as buffers of 32 MB hold, or, below the 8,192 rows from which on one kernel takes any number of them, the 4,096 rows of the
    # kernel for small batches: calls of critic.batch rows are short and many (65,600 rows: 33 of 11 us).
    width = critic.tick.shape[1]
    chunk = max(critic.batch, min(n, max(1, (1 << 23) // width)) if n >= 8192 else min(n, 4096))
    work = critic.__dict__.setdefault("_values_work", {})
    if work.get("rows") != chunk:
        z = lambda: torch.empty((chunk, width), device=critic.device, dtype=torch.float32)
        work["bytes"] = lib().b200rl_mlp_forward_workspace_bytes(C.byref(critic.shape), chunk)
        work.update(rows=chunk, tick=z(), tock=z(), buffer=torch.empty(max(work["bytes"], 16), device=critic.device, dtype=torch.uint8))
    return work


def evaluate_values(critic, dataset, layout):
    """critic(all observations) -> value column, as the PPO loop does before the advantage estimate
    (rl/algorithms/ppo/loop/core/operations_generic.h: evaluate(critic, all_observations_privileged, all_values))."""
    work = _values_work(critic, dataset.shape[0])
    n, chunk = dataset.shape[0], work["rows"]
    ld = dataset.stride(0)
    for begin in range(0, n, chunk):
        at = dataset.data_ptr() + 4 * begin * ld
        check(lib().b200rl_mlp_evaluate_ws(C.byref(critic.shape), _ptr(critic.params), at + 4 * layout.observations.start, ld, at + 4 * layout.values, ld, _ptr(work["tick"]),
                                           _ptr(work["tock"]), min(chunk, n - begin), _ptr(work["buffer"]), work["bytes"], _stream()), "b200rl_mlp_evaluate")
    return dataset


def _minibatch_update(actor, critic, rows, layout, epsilon_clip=0.2, entropy_coefficient=0.01, advantage_epsilon=1e-8, normalize_advantage=True, learn_action_std=True):
    import torch
    obs = rows[:, layout.observations]
    # the critic's update does not depend on the actor's: it runs on a second stream (a parallel branch once captured in a CUDA graph)
    side = critic.__dict__.get("_side_stream") or critic.__dict__.setdefault("_side_stream", torch.cuda.Stream(device=obs.device))
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        critic.zero_gradient()
        values = critic.forward(obs)
        critic.backward(obs, _mse_gradient(values, rows[:, layout.target_values:layout.target_values + 1], 0.5, d_a=critic.d_out_buffer()))
        critic.step()
    actor.zero_gradient()
    current = actor.forward(obs)
    d_actions = _ppo_policy_gradient(current, rows[:, layout.actions], actor.extra("params"), rows[:, layout.action_log_probs], rows[:, layout.advantages],
                                     actor.extra("grads"), epsilon_clip, entropy_coefficient, advantage_epsilon, normalize_advantage, learn_action_std,
                                     d_actions=actor.d_out_buffer(), scratch=actor.__dict__.setdefault("_ppo_scratch", {}))
    actor.backward(obs, d_actions)
    actor.step()
    torch.cuda.current_stream().wait_stream(side)


class MinibatchGraphs:
    """What `train` needs for one (actor, critic, dataset, batch_size) combination, made before its first call: scratch and shuffle buffers, and for networks that
    the one-launch epoch does not take one captured CUDA graph per minibatch position of the dataset matrix: the ~24 launches of a minibatch update
    replayed with a single launch. Every pointer is baked into the graphs. Should the epoch decline networks that it takes in general, they are captured then."""

    def __init__(self, actor, critic, dataset, layout, n_rows, batch_size, **hyper):
        self.key = (dataset.data_ptr(), n_rows, batch_size)
        self.graphs = []
        self._capture_arguments = (actor, critic, dataset, layout, n_rows, batch_size, hyper)
        _values_work(critic, dataset.shape[0])
        _shuffle(actor, dataset, layout, n_rows)
        if not _epoch_scratch(actor, critic, dataset, n_rows // batch_size, batch_size)["bytes"]:
            self._capture()

    def replay(self, b):
        if not self.graphs:
            self._capture()
        self.graphs[b].replay()

    def _capture(self):
        import torch
        actor, critic, dataset, layout, n_rows, batch_size, hyper = self._capture_arguments
        side = torch.cuda.Stream()
        side.wait_stream(torch.cuda.current_stream())
        saved = [t.clone() for t in (actor.params, actor.m, actor.v, actor.adam_state, critic.params, critic.m, critic.v, critic.adam_state)]
        with torch.cuda.stream(side):
            _minibatch_update(actor, critic, dataset[:batch_size], layout, **hyper)             # warm-up outside capture (lazy module loading)
        torch.cuda.current_stream().wait_stream(side)
        for b in range(n_rows // batch_size):
            g = torch.cuda.CUDAGraph()
            with torch.cuda.graph(g, stream=side):
                _minibatch_update(actor, critic, dataset[b * batch_size:(b + 1) * batch_size], layout, **hyper)
            self.graphs.append(g)
        for t, s in zip((actor.params, actor.m, actor.v, actor.adam_state, critic.params, critic.m, critic.v, critic.adam_state), saved):
            t.copy_(s)                                                                          # the warm-up update is undone


def _epoch_scratch(actor, critic, dataset, n_minibatches, batch_size):
    """Scratch of the one-launch epoch, kept with the actor; "bytes" is 0 for networks that its kernel does not take."""
    import torch
    work = actor.__dict__.setdefault("_epoch_scratch", {})
    key = (n_minibatches, batch_size, bytes(actor.shape), bytes(critic.shape))
    if work.get("key") != key:
        n = lib().b200rl_ppo_train_epoch_scratch_bytes(C.byref(actor.shape), C.byref(critic.shape), batch_size, n_minibatches)
        work["key"], work["bytes"], work["buffer"] = key, n, torch.empty(n, device=dataset.device, dtype=torch.uint8) if n else None
    return work


def _epoch_call(actor, critic, dataset, layout, n_minibatches, batch_size, epsilon_clip, entropy_coefficient, advantage_epsilon, normalize_advantage, learn_action_std):
    """All minibatch updates of one epoch as one native call: a function that issues it, made once per train() (an epoch of small networks takes 100 us);
    None for networks that its kernel does not take."""
    work = _epoch_scratch(actor, critic, dataset, n_minibatches, batch_size)
    if not work["bytes"]:
        return None
    base, ld = dataset.data_ptr(), dataset.stride(0)
    at = lambda column: base + 4 * column
    args = (C.byref(actor.shape), C.byref(actor.arenas()), C.byref(critic.shape), C.byref(critic.arenas()), at(layout.observations.start), at(layout.actions.start),
            at(layout.action_log_probs), at(layout.advantages), at(layout.target_values), ld, batch_size, n_minibatches, epsilon_clip, entropy_coefficient, advantage_epsilon,
            normalize_advantage, learn_action_std, work["buffer"].data_ptr(), work["bytes"], _stream())
    call = lib().b200rl_ppo_train_epoch

    def epoch():
        rc = call(*args)
        if rc == 2:                                                     # B200RL_ERR_UNSUPPORTED
            return False
        check(rc, "b200rl_ppo_train_epoch")
        return True
    return epoch


class _Shuffle:
    """The epoch shuffle: the next epoch's permutation is drawn and sent, on a stream of its own and into the other of two buffers, while this one's kernels
    run (a copy in the stream of the kernels held the epoch up by 25 to 40 us). Both pairs of buffers, device and pinned, are kept: the host draws into a
    pinned one once the copy out of it, two epochs before, has completed. An epoch is one native call."""

    def __init__(self, dataset, n_rows, columns):
        import torch
        self.n_rows, self.epoch = n_rows, 0
        self.scratch = _permute_rows_scratch(dataset, n_rows, columns)
        self.perm = torch.empty((2, n_rows), device=dataset.device, dtype=torch.int32)
        self.host = torch.empty((2, n_rows), dtype=torch.int32, pin_memory=True)
        self.stream = torch.cuda.Stream(device=dataset.device)
        self.used = [torch.cuda.current_stream().record_event() for _ in range(2)]
        self.sent = [self.stream.record_event() for _ in range(2)]

    def __call__(self, dataset, rng_state):
        k = self.epoch & 1
        mask, scratch, nbytes = self.scratch
        check(lib().b200rl_shuffle_rows(dataset.data_ptr(), dataset.stride(0), self.n_rows, mask, rng_state.ctypes.data, self.host[k].data_ptr(), self.perm[k].data_ptr(),
                                        scratch.data_ptr(), nbytes, self.sent[k].cuda_event, self.used[k].cuda_event, self.stream.cuda_stream, _stream()), "b200rl_shuffle_rows")
        self.epoch += 1


def _shuffle(actor, dataset, layout, n_rows):
    """The shuffle of the columns that an update reads, kept with the actor."""
    columns = list(range(layout.observations.start, layout.observations.stop)) + list(range(layout.actions.start, layout.actions.stop)) + \
        [layout.action_log_probs, layout.advantages, layout.target_values]
    key, work = (dataset.device, n_rows, tuple(columns)), actor.__dict__.setdefault("_shuffle", {})
    if key not in work:
        work.clear()
        work[key] = _Shuffle(dataset, n_rows, columns)
    return work[key]


def _train_epoch(*networks_and_sizes, **hyper):
    epoch = _epoch_call(*networks_and_sizes, **hyper)
    return epoch is not None and epoch()


def train(actor, critic, dataset, layout, n_rows, batch_size, n_epochs=10, epsilon_clip=0.2, entropy_coefficient=0.01, advantage_epsilon=1e-8,
          normalize_advantage=True, learn_action_std=True, shuffle_rng_state=None, graphs=None):
    """n_epochs x (n_rows // batch_size) minibatch updates. shuffle_rng_state (from rng_init_host) switches the reference's SHUFFLE_EPOCH
    on: before every epoch the observation / action / log-prob / advantage / target-value columns of the dataset matrix are permuted in
    place with the permutation the reference's engine would produce (:127-158); None keeps dataset order. Per minibatch: zero_gradient,
    actor forward, clipped-surrogate gradient (+ log_std gradient), actor backward, critic forward, 0.5-weighted MSE gradient against
    the target values, critic backward, one Adam step each. `actor` is an Mlp with extra_params = action_dim (the log_std behind the
    layers), `critic` an Mlp with one output; both built for batch_size rows. An epoch is one native call where its kernel takes the networks
    (small ones: up to three layers and about 18,000 parameters); otherwise graphs = a MinibatchGraphs built for these arguments replays each
    minibatch update as one CUDA graph launch instead of ~24 kernel launches (same kernels, same results)."""
    assert actor.batch == batch_size and critic.batch == batch_size and actor.n_extra == layout.action_dim
    hyper = dict(epsilon_clip=epsilon_clip, entropy_coefficient=entropy_coefficient, advantage_epsilon=advantage_epsilon,
                 normalize_advantage=normalize_advantage, learn_action_std=learn_action_std)
    if graphs is not None:
        assert graphs.key == (dataset.data_ptr(), n_rows, batch_size), "graphs were captured for another dataset matrix"
    epoch = _epoch_call(actor, critic, dataset, layout, n_rows // batch_size, batch_size, **hyper)
    shuffle = _shuffle(actor, dataset, layout, n_rows) if shuffle_rng_state is not None else None
    for _ in range(n_epochs):
        if shuffle is not None:
            shuffle(dataset, shuffle_rng_state)
        if epoch is not None and epoch():
            continue
        for b in range(n_rows // batch_size):
            if graphs is not None:
                graphs.replay(b)
            else:
                _minibatch_update(actor, critic, dataset[b * batch_size:(b + 1) * batch_size], layout, **hyper)
